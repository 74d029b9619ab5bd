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


def _run(wl, modes, chunks, learning=None):
    from visual_cortex_gb300 import _native as N
    from visual_cortex_gb300.model import Simulation
    sim = Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)
    try:
        if learning is not None:
            sim.set_ff_learning(learning)
        sim.set_record(N.REC_SPIKES, sum(chunks) + 1)
        for k, n in enumerate(chunks):
            want = modes[k % len(modes)]
            assert sim.persistent(int(want)) == (want and learning is None)
            sim.run(n)
        out = {"raster": sim.fetch_spikes(0, sum(chunks))}
        for s in ("v", "w", "gE", "hE", "gI", "hI", "gFF", "hFF", "tBack", "dep"):
            out[s] = sim.state(s)
        if learning is not None:
            for s in ("sLGN", "ff_post", "ff_pre", "total_ff"):
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


@pytest.mark.parametrize("mode,homeo,name", [(1, 0, "no_far"), (2, 2, "no_far"), (3, 1, "far"), (4, 1, "no_far"),
                                             (3, 2, "noise_failure")])
def test_plasticity_in_the_persistent_kernel(native, mode, homeo, name):
    """LGN->V1 learning, which runs in the same kernel where blocks are independent (not as the cooperative
    mode the plan reports): weights, post and presynaptic traces and homeostasis totals as the per-step
    kernel leaves them, also when the two take turns."""
    from visual_cortex_gb300.model import FFLearning
    learning = FFLearning(tauLTP=16.8, tauLTD=33.7, tauTrip=114.0, tauAvg=1000.0, targetFR=8.0 if mode == 1 else 0.0,
                          A_LGN=0.02, r_LTD=1.0, gmaxLGN=0.6, gminLGN=0.0, sRatioLGN=1.0, decayTimeHomeoFF=250.0,
                          applyHomeo=homeo, learning=mode, nLearnTypeFF_I=1 if mode == 2 else 0, tauLTP_I=16.8,
                          tauLTD_I=33.7, tauTrip_I=114.0, tauAvg_I=1000.0, A_LGN_I=0.01, r_LTD_I=1.0, gmaxLGN_I=0.6,
                          gminLGN_I=0.0, sRatioLGN_I=1.0, tauAvgCortical=500.0)
    wl = _workload(name)
    chunks = [65, 1, 70, 64]
    ref = _run(wl, [False], chunks, learning)
    assert np.abs(ref["sLGN"] - np.asarray(wl.net.sLGN, np.float32).ravel()).max() > (1e-4 if mode != 4 else -1)
    _same(ref, _run(wl, [True], chunks, learning))
    _same(ref, _run(wl, [True, False], chunks, learning))


@pytest.mark.parametrize("n,nblock,dur", [(22, 2, (5.0, 20.0)), (2, 3, (4.0, 9.0))])
def test_sweep_with_push_warps(native, n, nblock, dur):
    """Trials with far synapses take turns on the slots of the kernel with push warps (one CTA per SM), or have
    one each: every trial ends as it does alone."""
    from visual_cortex_gb300 import synth
    from visual_cortex_gb300.batch import Batch
    from visual_cortex_gb300.model import Simulation
    trials = synth.batch_trials(n_trials=n, nblock=nblock, n_lgn=512, width=64, height=64, nFrame=60, far_partners=60,
                                dur_ms=dur, seed=3)
    make = lambda wl: Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)
    batched = [make(tr.wl) for tr in trials]
    try:
        b = Batch(batched, [tr.steps for tr in trials], autotune=False)
        try:
            if n < 8:
                b.run(max_steps=20)
            assert b.sweep() > 0
        finally:
            b.close()
        for q, tr in enumerate(trials):
            alone = make(tr.wl)
            try:
                alone.persistent(0)
                alone.run(tr.steps)
                for k in ("v", "w", "tBack", "gE", "hE", "gI", "hI", "gFF", "hFF"):
                    np.testing.assert_array_equal(batched[q].state(k), alone.state(k), err_msg=f"trial {q} {k}")
            finally:
                alone.close()
    finally:
        for s in batched:
            s.close()
