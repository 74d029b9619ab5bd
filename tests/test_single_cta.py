"""Patches of one CTA with delayed synapses: no grid barrier separates the steps of the persistent kernel, only
the CTA's own."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(blockSize, nE, noDelay):
    from visual_cortex_gb300 import synth
    wl = synth.make_workload("one", seed=21, nblock=1, blockSize=blockSize, nE=nE, n_lgn=512, m=20, width=64, height=64,
                             nt=400, adex_inh=True, nFrame=40, wFF=0.35, noDelay=noDelay)
    if noDelay:   # far synapses: every neuron hears 30 others of its block after up to 1.5 ms
        rng = np.random.default_rng(3)
        n = wl.spec.nV1
        wl.net = dataclasses.replace(
            wl.net, nVec=np.full(n, 30, np.uint32), vecID=rng.integers(0, n, 30 * n).astype(np.uint32),
            conVec=rng.uniform(0.0, 0.01, 30 * n).astype(np.float32),
            delayVec=rng.uniform(0.02, 1.5, 30 * n).astype(np.float32))
    return wl


def _run(wl, modes, chunks):
    from visual_cortex_gb300 import _native as N
    from visual_cortex_gb300.model import Simulation
    sim = Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)
    try:
        sim.set_record(N.REC_SPIKES, sum(chunks) + 1)
        for k, n in enumerate(chunks):
            want = modes[k % len(modes)]
            assert sim.persistent(int(want)) == want
            sim.run(n)
        out = {s: sim.state(s) for s in ("v", "w", "gE", "hE", "gI", "hI", "gFF", "hFF", "tBack")}
        out["raster"] = sim.fetch_spikes(0, sum(chunks))
    finally:
        sim.close()
    return out


@pytest.mark.parametrize("blockSize,nE,noDelay", [(256, 192, 1), (96, 64, 1), (256, 192, 0)])
def test_one_cta_with_delayed_synapses(native, blockSize, nE, noDelay):
    wl = _workload(blockSize, nE, noDelay)
    chunks = [1, 64, 65, 2, 130]
    ref = _run(wl, [False], chunks)
    assert (ref["raster"] >= 1).sum() > 50
    for modes in ([True], [True, False]):
        got = _run(wl, modes, chunks)
        for k in ref:
            np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
