"""Batches on bitmask rows (what a batch falls back to where entry lists would not fit): both CTA sizes, rows resident in
shared memory and streamed, against the oracle and one another."""
import numpy as np
import pytest

from helpers import CONF, TOL_VSOMA_MV, hetero_state
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# one CTA and several, rows that fit in shared memory beside a second CTA, alone, and not at all
SIZES = [1, 33, 300, 1024, 1100, 2100, 5000]
DENS = [1.0, 0.5, 0.05, 0.3, 0.45, 0.12, 0.06]
STEPS = 300


@pytest.fixture(scope="module")
def ig(built):
    import infoli_gb300

    assert infoli_gb300.device_count() >= 1
    return infoli_gb300


@pytest.mark.parametrize("kahan", [False, True])
def test_bitmask_rows_match_the_oracle_in_every_layout(ig, kahan, monkeypatch):
    monkeypatch.setenv("INFOLI_BATCH_ROWS", "bits")
    conf = O.read_parameters(CONF)
    nets = [(n, ig.gen_bitmask(n, p, 5 + n), 0.03) for n, p in zip(SIZES, DENS)]
    states = [hetero_state(conf, n, 100 + n) for n in SIZES]
    first = None
    for block in (1024, 512):
        for residency in (ig.capi.RES_FIT, ig.capi.RES_OCC, ig.capi.RES_NONE):
            with ig.Batch(conf, nets, init_state=np.concatenate(states, axis=1), kahan=kahan, shape=block,
                          residency=residency) as bt:
                bt.set_stimulus_pulse(50, 100, 1.0)
                bt.run(STEPS)
                got, offsets = bt.get_state(), bt.offsets
            assert first is None or np.array_equal(got, first)  # the layout changes no result
            first = got
    monkeypatch.delenv("INFOLI_BATCH_ROWS")
    with ig.Batch(conf, nets, init_state=np.concatenate(states, axis=1), kahan=kahan) as bt:
        bt.set_stimulus_pulse(50, 100, 1.0)
        bt.run(STEPS)
        assert not np.array_equal(bt.get_state(), first)  # the lists sum in another order: that was the other kernel
    for i, (n, bits, g) in enumerate(nets):
        s = states[i].copy()
        O.run(n, conf[:23], s, *ig.bitmask_to_csr(n, bits), g_uniform=g, stim=("pulse", 50, 100, 1.0), nsteps=STEPS,
              trace_every=0, traces=("soma",), nthreads=O.max_threads())
        mine = first[:, offsets[i]:offsets[i + 1]]
        assert np.max(np.abs(mine[O.S["V_soma"]] - s[O.S["V_soma"]])) <= TOL_VSOMA_MV
        assert np.max(np.abs(mine[O.S["V_dend"]] - s[O.S["V_dend"]])) <= TOL_VSOMA_MV


@pytest.mark.parametrize("rows", ["lists", "bits"])
def test_autotune_times_each_layout_once(ig, rows, monkeypatch):
    """Entry lists have no residency: candidates that differ in it alone are one layout with one time."""
    if rows == "bits":
        monkeypatch.setenv("INFOLI_BATCH_ROWS", "bits")
    conf = O.read_parameters(CONF)
    nets = [(n, ig.gen_bitmask(n, p, 5 + n), 0.03) for n, p in zip(SIZES, DENS)]
    with ig.Batch(conf, nets, init_values=O.default_state(1, conf)[:, 0], shape="auto", tune_steps=20) as bt:
        ms = bt.tune["ms_per_step"]
        assert all(v > 0 for v in ms.values())
        assert ms[f"{bt.tune['block']}/{bt.tune['residency']}"] * 0.98 <= min(ms.values())
        if rows == "lists":
            assert ms["1024/none"] == ms["1024/fit"] and ms["512/none"] == ms["512/occupancy"] == ms["512/fit"]
            assert bt.tune["residency"] == "fit"
        bt.run(10)
