"""The persistent V1 kernel against the per-step kernel at the shapes where its paths change.

Both run the same float operations in the same order, so the spike words of every step and the
final state are equal bit for bit: blocks of one to four CTAs (the cluster of a block), a last CTA
with one active warp, networks without far synapses (no grid barrier) and with them (push warps),
near lists of a foreign block (spikes through global memory), runs of one step and of the chunk
length plus and minus one, and runs that hand over from one kernel to the other between chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "one_cta": dict(nblock=3, blockSize=256, nE=192, far_partners=40),
    "last_warp": dict(nblock=2, blockSize=544, nE=416, far_partners=40),
    "no_far": dict(nblock=2, blockSize=1024, nE=768),
    "far": dict(nblock=4, blockSize=1024, nE=768, far_partners=200),
    "noise_failure": dict(nblock=2, blockSize=640, nE=512, noisyDep=(0.2, 0.2), synFail=(0.1, 0.1, 0.1, 0.1),
                          synFailFF=(0.1, 0.1)),
    "delayed_near": dict(nblock=2, blockSize=512, nE=384, noDelay=0),
}


def _workload(name):
    from visual_cortex_gb300 import synth
    kw = dict(n_lgn=512, m=20, width=64, height=64, nt=400, adex_inh=True, nFrame=40, wFF=0.35)
    kw.update(CASES[name])
    return synth.make_workload(name, seed=31, **kw)


def _foreign(wl):
    """Every block also lists its neighbour, whose spikers reach it through half the own weights."""
    net, nb = wl.net, wl.spec.nblock
    net.nbId = np.stack([np.arange(nb), (np.arange(nb) + 1) % nb], 1).astype(np.uint32)
    net.nNearNB = np.full(nb, 2, np.uint32)
    net.conMat = np.concatenate([net.conMat, 0.5 * net.conMat], axis=1).astype(np.float32)
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
        out = {"raster": sim.fetch_spikes(0, sum(chunks))}
        for s in ("v", "w", "gE", "hE", "gI", "hI", "gFF", "hFF", "tBack", "dep"):
            out[s] = sim.state(s)
    finally:
        sim.close()
    return out


def _same(a, b):
    assert (a["raster"] >= 1).sum() > 50
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("name", sorted(CASES))
def test_persistent_equals_per_step(native, name):
    wl = _workload(name)
    chunks = [1, 63, 65, 2, 129]
    ref = _run(wl, [False], chunks)
    _same(ref, _run(wl, [True], chunks))


@pytest.mark.parametrize("name", ["far", "one_cta", "delayed_near"])
def test_kernels_hand_over_between_chunks(native, name):
    wl = _workload(name)
    chunks = [70, 1, 70, 1, 65, 30]
    _same(_run(wl, [False], chunks), _run(wl, [True, False], chunks))


@pytest.mark.parametrize("far", [0, 60])
def test_foreign_near_blocks(native, far):
    from visual_cortex_gb300 import synth
    wl = _foreign(synth.make_workload("foreign", seed=33, nblock=3, blockSize=640, nE=512, n_lgn=512, m=20, width=64,
                                      height=64, nt=400, adex_inh=True, nFrame=40, wFF=0.35, far_partners=far))
    chunks = [65, 1, 100]
    _same(_run(wl, [False], chunks), _run(wl, [True], chunks))
