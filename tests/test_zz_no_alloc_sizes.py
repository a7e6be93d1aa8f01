"""infoli_run_noalloc over its range of sizes against the float oracle: from many lanes per receiver to the fewest, one
pass over a CTA's receivers and several, rows of uneven length and none, the largest network that it takes."""
import ctypes as C

import numpy as np
import pytest

from helpers import CONF, TOL_VSOMA_MV, hetero_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(built):
    import torch

    import infoli_gb300 as ig

    assert ig.device_count() >= 1
    return ig, torch, O.read_parameters(CONF)


# cells per CTA and lanes per receiver on 152 SMs: 32 x 16, 33 x 8, 66 x 4, 129 x 4 (two passes), 432 x 4 (four)
@pytest.mark.parametrize("n", [1, 4864, 5003, 10001, 19600, 65536])
@pytest.mark.parametrize("per_edge_g", [False, True])
def test_noalloc_sizes_match_oracle(env, n, per_edge_g):
    ig, torch, conf = env
    rng, steps = np.random.default_rng(n), 60
    deg = np.minimum(rng.choice([0, 1, 7, 33, 70], n), n - 1)  # ragged: shorter and longer than a lane's loads
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    g = rng.uniform(0.005, 0.015, rp[-1]).astype(np.float32) if per_edge_g else None
    st0 = hetero_state(conf, n, 4)
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())  # noqa: E731
    d_rp, d_col, d_g, d_state = dev(rp), dev(col), dev(g), dev(st0.reshape(-1))
    d_tr = torch.zeros(steps * n, device="cuda")
    params, lib = np.ascontiguousarray(conf[:23], np.float32), ig.capi.load()
    rc = lib.infoli_run_noalloc(params.ctypes.data_as(C.c_void_p), n, ptr(d_rp), ptr(d_col), ptr(d_g), 0.01, 10, 40, 1.0,
                                ptr(d_state), 0, steps, ptr(d_tr), None)
    assert rc == 0, lib.infoli_last_error()
    want = st0.copy()
    ref = O.run(n, conf[:23], want, rp, col, g=g, g_uniform=0.01, stim=("pulse", 10, 40, 1.0), nsteps=steps,
                trace_every=1, traces=("axon",), nthreads=O.max_threads())["axon"]
    state = d_state.cpu().numpy().reshape(19, n)
    assert np.max(np.abs(state[O.S["V_soma"]] - want[O.S["V_soma"]])) <= TOL_VSOMA_MV
    assert np.max(np.abs(state[O.S["V_dend"]] - want[O.S["V_dend"]])) <= TOL_VSOMA_MV
    assert np.max(np.abs(d_tr.cpu().numpy().reshape(steps, n) - ref)) <= 10 * TOL_VSOMA_MV
    assert np.allclose(state, want, rtol=1e-3, atol=1e-3)
