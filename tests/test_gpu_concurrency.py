"""What one handle's calls may wait for: its own work, not the launches of others that leave SMs free."""
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


@pytest.fixture
def busy(ig):
    """A simulation of a few CTAs with about two seconds of steps enqueued."""
    conf, n = O.read_parameters(CONF), 50
    rp, col = ig.gen_uniform(n, 0.3, 2)
    with ig.Simulation(n, conf, rp, col, init_state=hetero_state(conf, n, 3)) as sim:
        sim.run(10)
        with _small(ig) as other:  # a kernel's first use loads it, which waits for the device
            other.run(20)
            other.get_state()
        sim.launch(1_500_000)
        yield sim
        sim.sync()


def _small(ig, n=50):
    conf = O.read_parameters(CONF)
    rp, col = ig.gen_uniform(n, 0.3, 4) if n > 2 else ig.gen_uniform(n, 1.0, 4)
    return ig.Simulation(n, conf, rp, col, init_state=hetero_state(conf, n, 5))


def test_create_run_and_destroy_beside_a_running_simulation(ig, busy):
    sim = _small(ig)
    sim.run(20)
    sim.get_state()
    sim.close()
    assert not busy.query()


def test_more_handles_than_error_words(ig, monkeypatch):
    sims = [_small(ig, 2) for _ in range(1030)]
    want = None
    for sim in sims:
        sim.run(3)
        got = sim.get_state()
        assert want is None or np.array_equal(got, want)
        want = got
    monkeypatch.setenv("INFOLI_STALL_CTA", "1")
    monkeypatch.setenv("INFOLI_WAIT_TIMEOUT_MS", "100")
    with _small(ig, 500) as last:  # without a word of its own: errors come from the device's
        with pytest.raises(ig.InfoliError) as e:
            last.run(5)
        assert e.value.code == ig.capi.ERR_TIMEOUT
    for sim in sims:
        sim.close()
    with _small(ig, 500) as again:
        with pytest.raises(ig.InfoliError) as e:
            again.run(5)
        assert e.value.code == ig.capi.ERR_TIMEOUT


def _batch(ig):
    conf = O.read_parameters(CONF)
    nets = [(n, ig.gen_bitmask(n, 0.2, n), 0.03) for n in (300, 1500)]
    return ig.Batch(conf, nets, init_state=hetero_state(conf, 1800, 3))


def test_batch_create_beside_a_running_simulation(ig):
    conf, n = O.read_parameters(CONF), 50
    rp, col = ig.gen_uniform(n, 0.3, 2)
    with _batch(ig) as first, ig.Simulation(n, conf, rp, col, init_state=hetero_state(conf, n, 3)) as busy:
        first.run(30)
        busy.run(10)
        busy.launch(1_500_000)
        second = _batch(ig)
        assert not busy.query()
        busy.sync()
        second.run(30)
        assert np.array_equal(second.get_state(), first.get_state())
        second.close()


def _noalloc(ig, torch, n, steps):
    """A call of the allocation-free run: its state after `steps` steps."""
    import ctypes as C

    conf = O.read_parameters(CONF)
    rp, col, g = ig.gen_fixed_degree(n, 30, 4, (0.02, 0.06))
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rp, col, g, hetero_state(conf, n, 5).reshape(-1))]
    torch.cuda.synchronize()
    ptr = [C.c_void_p(t.data_ptr()) for t in dev]
    side = torch.cuda.Stream()
    params, lib = np.ascontiguousarray(conf[:23], np.float32), ig.capi.load()

    def call():
        rc = lib.infoli_run_noalloc(params.ctypes.data_as(C.c_void_p), n, ptr[0], ptr[1], ptr[2], 0.04, 0, 0, 0.0, ptr[3], 0,
                                    steps, None, C.c_void_p(side.cuda_stream))
        assert rc == 0, lib.infoli_last_error()
        return dev[3].cpu().numpy()

    return call


@pytest.mark.parametrize("sms,ctas", [(76, None), (140, "10")])
def test_noalloc_beside_a_running_simulation(ig, sms, ctas, monkeypatch):
    """On half of the SMs it runs as it is, on a dozen with as few CTAs as its cells need."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count < 152:
        pytest.skip("sized for 152 SMs")
    if ctas:
        monkeypatch.setenv("INFOLI_NOALLOC_CTAS", ctas)
    conf, n = O.read_parameters(CONF), 10000
    call, again = _noalloc(ig, torch, 5003, 100), _noalloc(ig, torch, 5003, 100)
    want = call()
    rp, col = ig.gen_grid_gaussian(100, 100, 10.0, 18.0, 3)
    with ig.Simulation(n, conf, rp, col, init_state=hetero_state(conf, n, 3), grid=sms) as busy:
        assert busy.plan_info()["grid"] == sms
        busy.run(10)
        busy.launch(300_000)
        lib_done = again()
        assert not busy.query()
        busy.sync()
    assert np.array_equal(lib_done, want)
