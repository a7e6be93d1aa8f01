"""Infinite voltages (a simulation that has diverged): every state of the step is a number, an infinity or NaN where it
is in the oracle, which divides where the device multiplies by a reciprocal in two parts."""
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


@pytest.mark.parametrize("mode", ["stamped", "gather", "tgather", "bits", "stream"])
def test_infinite_voltages(ig, mode, monkeypatch):
    monkeypatch.setenv("INFOLI_SYNC", mode)
    conf, cases = O.read_parameters(CONF), [(v, x) for v in ("V_dend", "V_soma", "V_axon") for x in (np.inf, -np.inf)]
    n = len(cases) + 1
    st = O.default_state(n, conf)
    for c, (v, x) in enumerate(cases):  # the last cell stays as it is
        st[O.S[v], c] = x
    rp, col = np.zeros(n + 1, np.int64), np.zeros(0, np.int32)
    with ig.Simulation(n, conf, rp, col, init_state=st) as sim:
        sim.run(1)
        got = sim.get_state()
    want = st.copy()
    O.run(n, conf[:23], want, rp, col, g_uniform=conf[1], nsteps=1, trace_every=0, traces=())
    names = sorted(O.S, key=O.S.get)
    for f, name in enumerate(names):
        # the voltages and what the infinite one drives are infinite or NaN either way
        if name in ("V_dend", "V_soma", "V_axon", "I_CaH"):
            assert np.array_equal(np.isfinite(got[f]), np.isfinite(want[f])), name
            continue
        assert np.array_equal(np.isnan(got[f]), np.isnan(want[f])), (name, got[f], want[f])
        assert np.allclose(got[f], want[f], rtol=1e-5, atol=1e-7, equal_nan=True), (name, got[f], want[f])
