"""Stream plans on the GPU against the float oracle: cells per CTA from one to past the split of the gate units, one
and two sender shares (clusters), conductances per edge and uniform, launches split anywhere, and a stalled CTA."""
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


def _network(ig, n, edge_g):
    if n >= 2000:
        rp, col, g = ig.gen_fixed_degree(n, 20, 4, (0.02, 0.06))
    else:
        rp, col = ig.gen_uniform(n, 0.3 if n > 2 else 1.0, 2)
        g = np.random.default_rng(1).uniform(0.02, 0.06, len(col)).astype(np.float32)
    return rp, col, g if edge_g else None


@pytest.mark.parametrize("kahan,edge_g", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n,grid", [(1, "0"), (33, "1"), (600, "2"), (1025, "2"), (2500, "152"), (61001, "0")])
def test_stream_plans_match_oracle(ig, n, grid, kahan, edge_g, monkeypatch):
    conf = O.read_parameters(CONF)
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    if grid != "0":
        monkeypatch.setenv("INFOLI_GRID", grid)
    rp, col, g = _network(ig, n, edge_g)
    st0 = hetero_state(conf, n, 3)
    steps, rng = 40 if n > 10000 else 300, np.random.default_rng(5)
    amp, onset = rng.uniform(0, 3, n).astype(np.float32), rng.integers(0, steps, n).astype(np.int32)
    with ig.Simulation(n, conf, rp, col, g=g, init_state=st0, kahan=kahan) as sim:
        sim.set_stimulus_cells(amp, onset, 20)
        a, b = sim.run(steps // 3, 1, ig.TRACE_SOMA)["soma"], sim.run(steps - steps // 3, 1, ig.TRACE_SOMA)["soma"]
        got, state = np.concatenate([a, b]), sim.get_state()
    with ig.Simulation(n, conf, rp, col, g=g, init_state=st0, kahan=kahan) as sim:
        sim.set_stimulus_cells(amp, onset, 20)
        assert np.array_equal(got, sim.run(steps, 1, ig.TRACE_SOMA)["soma"])  # launch boundaries change nothing
        assert np.array_equal(state, sim.get_state())
    table = np.where((np.arange(steps)[:, None] >= onset) & (np.arange(steps)[:, None] < onset + 20), amp, 0)
    with ig.Simulation(n, conf, rp, col, g=g, init_state=st0, kahan=kahan) as sim:
        sim.set_stimulus_table(table.astype(np.float32), 0)
        assert np.array_equal(got, sim.run(steps, 1, ig.TRACE_SOMA)["soma"])
    # the oracle with the reference's pulse off (steps below 20,000) and a table in its place: the network's own currents
    monkeypatch.setenv("INFOLI_SYNC", "gather")
    monkeypatch.delenv("INFOLI_GRID", raising=False)
    with ig.Simulation(n, conf, rp, col, g=g, init_state=st0, kahan=kahan) as sim:
        sim.set_stimulus_cells(amp, onset, 20)
        other = sim.run(steps, 1, ig.TRACE_SOMA)["soma"]
    assert np.max(np.abs(got - other)) <= TOL_VSOMA_MV
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    with ig.Simulation(n, conf, rp, col, g=g, init_state=st0, kahan=kahan) as sim:
        mine = sim.run(steps, 1, ig.TRACE_SOMA)["soma"]
    st = st0.copy()
    ref = O.run(n, conf[:23], st, rp, col, g=g, g_uniform=conf[1], nsteps=steps, trace_every=1, traces=("soma",),
                nthreads=O.max_threads())["soma"]
    assert np.max(np.abs(mine - ref)) <= TOL_VSOMA_MV


@pytest.mark.parametrize("n", [2000, 61001])
def test_stalled_cta_times_out_and_recovers(ig, n, monkeypatch):
    conf = O.read_parameters(CONF)
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    monkeypatch.setenv("INFOLI_WAIT_TIMEOUT_MS", "300")
    rp, col, _ = _network(ig, n, False)
    st0 = hetero_state(conf, n, 2)
    with ig.Simulation(n, conf, rp, col, init_state=st0) as sim, ig.Simulation(n, conf, rp, col, init_state=st0) as ref:
        monkeypatch.setenv("INFOLI_STALL_CTA", "1")
        with pytest.raises(ig.InfoliError) as e:
            sim.run(50)
        assert e.value.code == ig.capi.ERR_TIMEOUT
        monkeypatch.delenv("INFOLI_STALL_CTA")
        sim.set_state(st0)
        a, b = ref.run(60, 1, ig.TRACE_SOMA)["soma"], sim.run(60, 1, ig.TRACE_SOMA)["soma"]
        assert np.isfinite(a).all() and np.array_equal(a, b)
