"""Stream plans whose launch gives up: every CTA of every cluster leaves on the same step, whichever CTA stalls, time
after time, and the handle goes on with a new state."""
import time

import numpy as np
import pytest

from helpers import CONF, hetero_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ig(built):
    import infoli_gb300

    assert infoli_gb300.device_count() >= 1
    return infoli_gb300


@pytest.mark.parametrize("n", [2000, 61001])  # one share of the senders, and two (clusters)
def test_stalls_end_in_a_timeout_wherever_and_however_often(ig, n, monkeypatch):
    conf = O.read_parameters(CONF)
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    monkeypatch.setenv("INFOLI_WAIT_TIMEOUT_MS", "100")
    rp, col, _ = ig.gen_fixed_degree(n, 20, 4, (0.02, 0.06))
    st0 = hetero_state(conf, n, 2)
    with ig.Simulation(n, conf, rp, col, init_state=st0) as sim:
        want = sim.run(30, 1, ig.TRACE_SOMA)["soma"]
        grid = sim.plan_info()["grid"]
        for cta in (0, 1, grid - 1, 0, grid // 2, 1):
            monkeypatch.setenv("INFOLI_STALL_CTA", str(cta))
            t0 = time.time()
            with pytest.raises(ig.InfoliError) as e:
                sim.run(50)
            assert e.value.code == ig.capi.ERR_TIMEOUT and time.time() - t0 < 10
        monkeypatch.delenv("INFOLI_STALL_CTA")
        sim.set_state(st0)
        assert np.array_equal(sim.run(30, 1, ig.TRACE_SOMA)["soma"], want)


@pytest.mark.parametrize("limit_ms", ["1", "3"])
def test_waits_that_run_out_early_leave_no_copies_behind(ig, limit_ms, monkeypatch):
    """Limits of a few hundred steps, so that waits run out at any point of a step; whatever the CTAs had under way, the
    launches after them (other kernels on the same shared memory among them) compute what they did before."""
    conf, n = O.read_parameters(CONF), 20000
    rp, col, _ = ig.gen_fixed_degree(n, 20, 4, (0.02, 0.06))
    rp2, col2 = ig.gen_uniform(900, 0.1, 2)
    st0, st2 = hetero_state(conf, n, 2), hetero_state(conf, 900, 3)
    monkeypatch.setenv("INFOLI_SYNC", "stream")
    with ig.Simulation(n, conf, rp, col, init_state=st0) as sim:
        want = sim.run(30, 1, ig.TRACE_SOMA)["soma"]
        monkeypatch.setenv("INFOLI_SYNC", "auto")
        with ig.Simulation(900, conf, rp2, col2, init_state=st2) as other:
            want2 = other.run(30, 1, ig.TRACE_SOMA)["soma"]
            for cta in range(0, 150, 10):
                monkeypatch.setenv("INFOLI_STALL_CTA", str(cta))
                monkeypatch.setenv("INFOLI_WAIT_TIMEOUT_MS", limit_ms)
                with pytest.raises(ig.InfoliError) as e:
                    sim.run(50)
                assert e.value.code == ig.capi.ERR_TIMEOUT
                monkeypatch.delenv("INFOLI_STALL_CTA")
                monkeypatch.delenv("INFOLI_WAIT_TIMEOUT_MS")
                other.set_state(st2)
                assert np.array_equal(other.run(30, 1, ig.TRACE_SOMA)["soma"], want2)
                sim.set_state(st0)
                assert np.array_equal(sim.run(30, 1, ig.TRACE_SOMA)["soma"], want)
