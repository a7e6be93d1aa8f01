"""The dealing of a stream plan's entries by shared-memory bank: every entry once (the emulated currents are right), and
with few conflicts, over lane-chunk lengths, one and several shares, senders that crowd a few banks, and repeats."""
import numpy as np
import pytest

from test_planner import capi, check  # noqa: F401

STREAM = 6


def _per_gather(info):
    return info["gather_wavefronts"] / max(1, info["gathers"])


@pytest.mark.parametrize("edge_g", [False, True])
@pytest.mark.parametrize("n,degree,most", [(3001, 900, 2.2), (6007, 1500, 1.8), (4000, 60, 2.6)])
def test_conflicts_are_few(capi, n, degree, most, edge_g):  # noqa: F811
    rng = np.random.default_rng(n)
    rp = np.arange(n + 1, dtype=np.int64) * degree
    col = np.concatenate([np.sort(rng.choice(n, degree, replace=False)) for _ in range(n)]).astype(np.int32)
    g = rng.uniform(0.02, 0.06, len(col)).astype(np.float32) if edge_g else None
    assert _per_gather(check(capi, n, rp, col, g=g, sync_mode=STREAM)) < most  # 3.5 in any order


@pytest.mark.parametrize("budget", [232448 - 1024, 9000])  # one share, and clusters
def test_crowded_banks_and_repeats(capi, budget):  # noqa: F811
    n, rng = 1990, np.random.default_rng(4)
    deg = rng.choice([0, 1, 3, 31, 32, 33, 64, 400], n)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    col = rng.integers(0, n, rp[-1])
    col = np.where(rng.random(len(col)) < 0.7, col // 32 * 32 + 5, col)  # most senders in one bank
    col = np.minimum(col, n - 1).astype(np.int32)
    g = rng.uniform(0.02, 0.06, len(col)).astype(np.float32)
    check(capi, n, rp, col, g=g, sync_mode=STREAM, smem_budget=budget)
    check(capi, n, rp, col, sync_mode=STREAM, smem_budget=budget)
