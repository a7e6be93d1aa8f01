"""Stream plans on the CPU: the emulated walk of their tables (every index checked, padding entries included) gives
the gap-junction currents of the CSR network, for one and several sender shares, ragged rows, duplicates of a sender,
self edges, empty rows and any sender order; and auto mode takes them where their rule says."""
import numpy as np
import pytest

from test_planner import capi, check  # noqa: F401

STREAM, STREAM_CODE = 6, 5


@pytest.mark.parametrize("grid", [0, 1, 7, 152])
@pytest.mark.parametrize("n,p", [(1, 0.5), (2, 1.0), (33, 1.0), (1000, 0.1), (3001, 0.3)])
def test_uniform_networks(capi, n, p, grid):  # noqa: F811
    rp, col = capi.gen_uniform(n, p, 1)
    info = check(capi, n, rp, col, sync_mode=STREAM, grid=grid)
    assert info["stamped"] == STREAM_CODE


# a budget that the whole V_dend array does not fit: shares over clusters of 2 and 4
@pytest.mark.parametrize("budget,cluster", [(7000, 2), (3800, 4)])
def test_sender_shares(capi, budget, cluster):  # noqa: F811
    n = 1999
    rp, col, g = capi.gen_fixed_degree(n, 25, 6, (0.02, 0.06))
    info = check(capi, n, rp, col, g=g, sync_mode=STREAM, smem_budget=budget)
    assert info["stamped"] == STREAM_CODE and info["ctas"] % cluster == 0


def test_ragged_rows_in_any_order(capi):  # noqa: F811
    n, rng = 700, np.random.default_rng(2)
    deg = np.where(rng.random(n) < 0.2, 0, rng.integers(0, 400, n))
    deg[5] = 3000  # longer than any cut of the others, repeated senders among them
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)  # unsorted, with repeats and self edges
    g = rng.uniform(0.02, 0.06, rp[-1]).astype(np.float32)
    for kw in (dict(), dict(grid=3), dict(g=g), dict(g=g, smem_budget=4200)):
        check(capi, n, rp, col, sync_mode=STREAM, **kw)


def test_auto_rule(capi):  # noqa: F811
    rp, col = capi.gen_bitmask_csr(9000, 0.2, 5)
    assert check(capi, 9000, rp, col)["stamped"] == STREAM_CODE
    rp, col = capi.gen_bitmask_csr(6000, 0.5, 5)  # dense enough for a bit per pair
    assert check(capi, 6000, rp, col)["stamped"] == 4
    rp, col, g = capi.gen_fixed_degree(70000, 20, 12, (0.02, 0.06))  # two shares
    info = check(capi, 70000, rp, col, g=g)
    assert info["stamped"] == STREAM_CODE and info["ctas"] == 152
