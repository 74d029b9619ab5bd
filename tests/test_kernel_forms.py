"""Which form of the V1 kernel a plan gets, and forms that only patches of certain sizes get.

The persistent launch tries a block's CTAs as a cluster with push warps (one CTA per SM), the cluster without them (two
CTAs per SM), single CTAs; per-step launches are the fallback of all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("v", "w", "gE", "hE", "gI", "hI", "gFF", "hFF", "tBack")


def _workload(**kw):
    from visual_cortex_gb300 import synth
    args = dict(n_lgn=512, m=20, width=64, height=64, nt=400, adex_inh=True, nFrame=40, wFF=0.35)
    args.update(kw)
    return synth.make_workload("form", seed=51, **args)


def _run(wl, mode, chunks, learning=None, state=STATE):
    from visual_cortex_gb300 import _native as N
    from visual_cortex_gb300.model import Simulation
    sim = Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)
    launches = []
    try:
        if learning is not None:
            sim.set_ff_learning(learning)
        sim.set_record(N.REC_SPIKES, sum(chunks) + 1)
        assert sim.persistent(int(mode)) == (mode and learning is None)
        for n in chunks:
            sim.run(n)
            launches.append(int(N.lib.pv1_last_launch_count(sim.plan)))
        out = {s: sim.state(s) for s in state}
        out["raster"] = sim.fetch_spikes(0, sum(chunks))
    finally:
        sim.close()
    return out, launches


def _same(a, b):
    assert (a["raster"] >= 1).sum() > 50
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("nblock,blockSize,nE", [
    (90, 288, 224),     # 180 CTAs: two per SM, in clusters of two
    (100, 520, 392),    # 300 CTAs of 304: not all of them in clusters of three, each CTA by itself
])
def test_patches_of_more_ctas_than_sms(native, nblock, blockSize, nE):
    wl = _workload(nblock=nblock, blockSize=blockSize, nE=nE, far_partners=12, wFar=0.01)
    chunks = [1, 64, 40]
    ref, many = _run(wl, False, chunks)
    got, few = _run(wl, True, chunks)
    assert many[1] >= 64 and few[1] < 16
    _same(ref, got)


def _learning(mode):
    from visual_cortex_gb300.model import FFLearning
    return FFLearning(tauLTP=16.8, tauLTD=33.7, tauTrip=114.0, tauAvg=1000.0, targetFR=8.0 if mode == 1 else 0.0,
                      A_LGN=0.02, r_LTD=1.0, gmaxLGN=0.6, gminLGN=0.0, sRatioLGN=1.0, decayTimeHomeoFF=250.0,
                      applyHomeo=1, learning=mode, nLearnTypeFF_I=1 if mode == 2 else 0, tauLTP_I=16.8, tauLTD_I=33.7,
                      tauTrip_I=114.0, tauAvg_I=1000.0, A_LGN_I=0.01, r_LTD_I=1.0, gmaxLGN_I=0.6, gminLGN_I=0.0,
                      sRatioLGN_I=1.0, tauAvgCortical=500.0)


@pytest.mark.parametrize("mode,shape,chunked", [
    (1, dict(nblock=2, blockSize=1024, nE=768), True),
    (2, dict(nblock=4, blockSize=224, nE=160), True),            # one CTA per block, partly filled
    (3, dict(nblock=2, blockSize=544, nE=416), True),            # a last CTA of one warp
    (4, dict(nblock=3, blockSize=256, nE=192), True),
    (3, dict(nblock=2, blockSize=512, nE=384, far_partners=40), False),   # blocks that are coupled
    (3, dict(nblock=2, blockSize=512, nE=384, noDelay=0), False),
])
def test_plasticity_takes_the_persistent_kernel(native, mode, shape, chunked):
    """Plans with plasticity report no persistent mode: the launches of a 64-step run tell."""
    wl = _workload(**shape)
    state = STATE + ("sLGN", "ff_post", "ff_pre", "total_ff")
    chunks = [1, 64, 70]
    ref, many = _run(wl, False, chunks, _learning(mode), state)
    got, few = _run(wl, True, chunks, _learning(mode), state)
    assert many[1] >= 64
    assert few[1] < 16 if chunked else few[1] >= 64
    _same(ref, got)
