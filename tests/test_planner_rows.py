"""Tile and stamped plans of networks whose rows are not in order: senders shuffled and repeated inside a row, rows of very uneven length.
The tables must hold what the ordered rows' tables hold (equal senders keep the caller's order)."""
import numpy as np
import pytest


@pytest.fixture(scope="module")
def capi(built):
    from infoli_gb300 import capi

    return capi


@pytest.mark.parametrize("per_edge_g", [False, True])
@pytest.mark.parametrize("mode,budget", [(1, 232448 - 1024), (1, 20000), (2, 232448 - 1024)])
def test_rows_in_any_order_give_the_same_plan(capi, mode, budget, per_edge_g):
    rng, n = np.random.default_rng(3), 3000
    lens = rng.choice([0, 1, 31, 32, 33, 200, 900], n)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)  # with repeats
    g = rng.uniform(0.01, 0.05, rp[-1]).astype(np.float32) if per_edge_g else None
    order = np.lexsort((np.arange(rp[-1]), col, np.repeat(np.arange(n), lens)))
    v = (-60 + rng.uniform(-15, 15, n)).astype(np.float32)
    kw = dict(sync_mode=mode, smem_budget=budget, threads=512)
    got, info = capi.plan_emulate(n, rp, col, v, g=g, **kw)
    want, same = capi.plan_emulate(n, rp, col[order], v, g=None if g is None else g[order], **kw)
    assert np.array_equal(got, want) and info == same
    V = v[np.repeat(np.arange(n), lens)].astype(np.float64) - v[col]
    exact = np.bincount(np.repeat(np.arange(n), lens), (0.04 if g is None else g) * (0.8 * np.exp(-V * V / 100) + 0.2) * V, n)
    assert np.max(np.abs(got - exact) / np.maximum(1.0, np.abs(exact))) < 2e-4
