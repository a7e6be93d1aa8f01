"""Stream plans take the differences of V_dend before anything is rounded: pairs of cells a few units in the last place
apart, coupled so strongly that a rounding of their voltages would show, one step against the FP64 oracle."""
import numpy as np
import pytest

from helpers import CONF
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ig(built):
    import infoli_gb300

    assert infoli_gb300.device_count() >= 1
    return infoli_gb300


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("edge_g", [False, True])
@pytest.mark.parametrize("n", [64, 62000])  # one share of the senders, and two
def test_small_differences_of_strongly_coupled_cells(ig, n, edge_g, kahan, monkeypatch):
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    conf, rng, g = O.read_parameters(CONF), np.random.default_rng(n), 1000.0
    st = O.default_state(n, conf)
    v = rng.uniform(-63, -33, n // 2).astype(np.float32)
    st[O.S["V_dend"], 0::2] = v
    st[O.S["V_dend"], 1::2] = v + rng.integers(1, 5, n // 2).astype(np.float32) * np.spacing(v)
    rp, col = np.arange(n + 1, dtype=np.int64), (np.arange(n, dtype=np.int32) ^ 1)  # each one's sender is its pair
    with ig.Simulation(n, conf, rp, col, g=np.full(n, g, np.float32) if edge_g else None, g_uniform=g, init_state=st,
                       kahan=kahan) as sim:
        sim.run(1)
        got = sim.get_state()[O.S["V_dend"]].astype(np.float64)
    want = st.astype(np.float64)
    O.run(n, conf[:23].astype(np.float64), want, rp, col, g_uniform=g, nsteps=1, trace_every=0, traces=(), fp64=True)
    # a term's relative error is about 1e-6 of at most 1,000 x 4 x 4e-6 x 0.05; the other currents' less: the new
    # voltage's own rounding and as much again.  A voltage scaled and rounded first is off by up to 4e-6 x 1,000 x 0.05
    assert np.max(np.abs(got - want[O.S["V_dend"]])) <= 4e-6
