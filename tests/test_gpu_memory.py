"""infoli_sim_memory against what a simulation takes from the device's pool: a server admits requests by this number."""
import ctypes

import pytest

from helpers import CONF
from oracle import oracle as O

pytestmark = pytest.mark.gpu

USED_NOW = 7  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT


@pytest.fixture(scope="module")
def ig(built):
    import infoli_gb300

    assert infoli_gb300.device_count() >= 1
    return infoli_gb300


def _used(ig):
    lib, cu, v = ig.capi.load(), ctypes.CDLL("libcuda.so.1"), ctypes.c_uint64(0)
    lib.infoli__device_pool.restype, lib.infoli__device_pool.argtypes = ctypes.c_void_p, [ctypes.c_int]
    assert cu.cuMemPoolGetAttribute(ctypes.c_void_p(lib.infoli__device_pool(0)), USED_NOW, ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("mode", ["stream", "tgather", "stamped", "auto"])
def test_memory_is_what_the_pool_gave(ig, mode, monkeypatch):
    conf, n = O.read_parameters(CONF), 40000 if mode == "stamped" else 100000
    monkeypatch.setenv("INFOLI_SYNC", mode)
    rp, col, _ = ig.gen_fixed_degree(n, 3 if mode == "stamped" else 20, 4, (0.02, 0.06))
    with ig.Simulation(n, conf, rp, col, init_values=O.default_state(1, conf)[:, 0]):
        pass  # the first one makes the pool
    before = _used(ig)
    with ig.Simulation(n, conf, rp, col, init_values=O.default_state(1, conf)[:, 0]) as sim:
        taken = _used(ig) - before
        said = sim.device_bytes()
    # some 20 allocations, each rounded up; an array of n floats would be 400 KB (160 KB)
    assert abs(taken - said) < 150000
