"""Stream plans over clusters of four CTAs (networks whose V_dend takes four shares) against the float oracle."""
import numpy as np
import pytest

from helpers import CONF, TOL_VSOMA_MV, hetero_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N, STEPS = 108001, 40


@pytest.fixture(scope="module")
def net(built):
    import infoli_gb300 as ig

    assert ig.device_count() >= 1
    conf = O.read_parameters(CONF)
    return ig, conf, ig.gen_fixed_degree(N, 20, 4, (0.02, 0.06)), hetero_state(conf, N, 3)


def _four_shares(sim):
    info = sim.plan_info()
    assert info["threads"] == 768 and info["grid"] % 4 == 0
    assert info["smem_bytes"] < 4 * (N // 2)  # half of V_dend is not there


@pytest.mark.parametrize("kahan", [False, True])
@pytest.mark.parametrize("edge_g", [False, True])
def test_four_shares_match_oracle(net, edge_g, kahan):
    ig, conf, (rp, col, g), st0 = net
    with ig.Simulation(N, conf, rp, col, g=g if edge_g else None, init_state=st0, kahan=kahan) as sim:
        _four_shares(sim)
        got = np.concatenate([sim.run(k, 1, ig.TRACE_SOMA)["soma"] for k in (1, STEPS - 1)])
    st = st0.copy()
    ref = O.run(N, conf[:23], st, rp, col, g=g if edge_g else None, g_uniform=conf[1], nsteps=STEPS, trace_every=1,
                traces=("soma",), nthreads=O.max_threads())["soma"]
    assert np.max(np.abs(got - ref)) <= TOL_VSOMA_MV


def test_stalls_in_clusters_of_four_end_in_a_timeout(net, monkeypatch):
    ig, conf, (rp, col, _), st0 = net
    monkeypatch.setenv("INFOLI_WAIT_TIMEOUT_MS", "100")
    with ig.Simulation(N, conf, rp, col, init_state=st0) as sim:
        _four_shares(sim)
        want = sim.run(20, 1, ig.TRACE_SOMA)["soma"]
        for cta in (0, 1, 2, 3, sim.plan_info()["grid"] - 1):
            monkeypatch.setenv("INFOLI_STALL_CTA", str(cta))
            with pytest.raises(ig.InfoliError) as e:
                sim.run(50)
            assert e.value.code == ig.capi.ERR_TIMEOUT
        monkeypatch.delenv("INFOLI_STALL_CTA")
        sim.set_state(st0)
        assert np.array_equal(sim.run(20, 1, ig.TRACE_SOMA)["soma"], want)
