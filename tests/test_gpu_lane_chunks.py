"""The stamped step kernel with lane-chunks of 8, 16 and 32 entries against the gather kernel."""
import numpy as np
import pytest

from helpers import CONF, TOL_VSOMA_MV, hetero_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ig(built):
    import infoli_gb300

    assert infoli_gb300.device_count() >= 1
    return infoli_gb300


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("per_edge_g", [False, True])
@pytest.mark.parametrize("n,lens", [(2, (1,)), (65, (7, 8, 9)), (1000, (31, 32)), (1000, (31, 33)), (700, (0, 100, 250)),
                                    (700, (600,))])
def test_lane_chunks_match_the_gather_kernel(ig, n, lens, per_edge_g, kahan, monkeypatch):
    conf, rng = O.read_parameters(CONF), np.random.default_rng(n)
    count = np.minimum(rng.choice(lens, n), n - 1)
    rp = np.concatenate([[0], np.cumsum(count)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in count]).astype(np.int32)
    g = rng.uniform(0.002, 0.006, rp[-1]).astype(np.float32) if per_edge_g else None
    got = {}
    for mode in ("stamped", "gather"):
        monkeypatch.setenv("INFOLI_SYNC", mode)
        with ig.Simulation(n, conf, rp, col, g=g, g_uniform=0.004, init_state=hetero_state(conf, n, 3), kahan=kahan) as sim:
            sim.set_stimulus_cells(np.full(n, 1.5, np.float32), np.arange(n, dtype=np.int32) % 90, 20)
            got[mode] = sim.run(200, 1, ig.TRACE_SOMA)["soma"]
    assert np.max(np.abs(got["stamped"] - got["gather"])) <= TOL_VSOMA_MV
