"""Lane-chunks of 8, 16 and 32 entries in stamped plans: the plan's tables hold the network at the edges of every rule
(rows around multiples of the chunk, groups around half of the warps), and the CTA's partial sums stay in order."""
import numpy as np
import pytest


@pytest.fixture(scope="module")
def capi(built):
    from infoli_gb300 import capi

    return capi


@pytest.mark.parametrize("per_edge_g", [False, True])
@pytest.mark.parametrize("n,lens,grid_max", [
    (1, (0,), 152), (2, (1,), 152), (50, (7, 8, 9), 152), (64, (31, 32), 152), (64, (31, 33), 152), (40, (15, 16, 17), 1),
    (85, (24,), 1), (86, (24,), 1), (64, (32,), 1), (65, (32,), 1), (32, (128,), 1), (33, (128,), 1), (500, (0, 40, 200), 152),
    (1400, (8, 60), 152), (1600, (8, 60), 152)])
def test_lane_chunk_tables_hold_the_network(capi, n, lens, grid_max, per_edge_g):
    rng = np.random.default_rng(n)
    count = np.minimum(rng.choice(lens, n), max(n - 1, 0) * 4)
    rp = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    g = rng.uniform(0.01, 0.05, rp[-1]).astype(np.float32) if per_edge_g else None
    v = (-60 + rng.uniform(-15, 15, n)).astype(np.float32)
    got, info = capi.plan_emulate(n, rp, col, v, g=g, sync_mode=2, threads=512, grid_max=grid_max)
    assert info["stamped"] == 1
    dst = np.repeat(np.arange(n), count)
    V = v[dst].astype(np.float64) - v[col]
    terms = (0.04 if g is None else g) * (0.8 * np.exp(-V * V / 100) + 0.2) * V
    want, size = np.bincount(dst, terms, n), np.bincount(dst, np.abs(terms), n)
    # float sums of up to 200 terms, exponential to 2 ulp: half an ulp per addition and a few per term
    assert np.all(np.abs(got - want) <= (np.maximum(count, 1) + 40) * 6e-8 * size + 1e-12)
