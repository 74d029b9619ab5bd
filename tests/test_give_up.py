"""Waits of the persistent V1 kernels that run out, in every form of the kernel: the run ends with PV1_E_DEVICE
(or, where no wait took that long, as it should), and the GPU goes on to run the next plan.

A limit of 0 polls makes each wait for the grid end before its first poll.  The others lie around what waits take
(a poll of the grid barrier is about 50 ns), so that CTAs of a block give up in different steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {
    "push_warps": dict(nblock=4, blockSize=1024, nE=768, far_partners=60),
    "two_ctas_per_sm": dict(nblock=90, blockSize=288, nE=224, far_partners=30),
    "one_cta_blocks": dict(nblock=6, blockSize=256, nE=192, far_partners=30),
    "independent_blocks": dict(nblock=3, blockSize=1024, nE=768),
    "delayed_near": dict(nblock=3, blockSize=512, nE=384, noDelay=0),
}


def _workload(name):
    from visual_cortex_gb300 import synth
    return synth.make_workload(name, seed=41, n_lgn=512, m=20, width=64, height=64, nt=400, adex_inh=True, nFrame=40,
                               wFF=0.35, **SHAPES[name])


def _sim(wl):
    from visual_cortex_gb300.model import Simulation
    return Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)


def _limited(native, wl, limit, steps, learning=None):
    sim = _sim(wl)
    try:
        if learning is not None:
            sim.set_ff_learning(learning)
        else:
            assert sim.persistent(1)
        native.check(sim.plan, native.lib.pv1_set_wait_limit(sim.plan, limit), "pv1_set_wait_limit")
        rc = native.lib.pv1_run(sim.plan, steps, 1)
        if rc == -5:
            assert "barrier wait gave up" in native.lib.pv1_last_error(sim.plan).decode()
        return rc, sim.state("v") if rc == 0 else None
    finally:
        sim.close()


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_limits(native, name):
    wl = _workload(name)
    steps = 70
    want = None
    for limit in (-1, 0, 1, 16, 128, 512, 2048, 8192, 32768, -1):
        rc, v = _limited(native, wl, limit, steps)
        assert rc in (0, -5), (limit, rc)
        if limit == 0:
            assert rc == -5
        if limit == -1:
            assert rc == 0
            want = v if want is None else want
        if rc == 0:
            np.testing.assert_array_equal(v, want, err_msg=f"limit {limit}")


def test_limits_with_plasticity(native):
    """Clusters without a grid barrier: only the waits for the block's spikes."""
    from visual_cortex_gb300.model import FFLearning
    learning = FFLearning(tauLTP=16.8, tauLTD=33.7, tauTrip=114.0, tauAvg=1000.0, targetFR=0.0, A_LGN=0.02, r_LTD=1.0,
                          gmaxLGN=0.6, gminLGN=0.0, sRatioLGN=1.0, decayTimeHomeoFF=250.0, applyHomeo=1, learning=3,
                          nLearnTypeFF_I=0, tauAvgCortical=500.0)
    wl = _workload("independent_blocks")
    want = None
    for limit in (-1, 0, 64, 128, 4096, -1):
        rc, v = _limited(native, wl, limit, 70, learning)
        assert rc in (0, -5), (limit, rc)
        if limit == -1:
            assert rc == 0
            want = v if want is None else want
        if rc == 0:
            np.testing.assert_array_equal(v, want, err_msg=f"limit {limit}")


@pytest.mark.parametrize("n", [3, 24])
def test_limits_in_a_batch(native, n):
    """The form with push warps (a slot per trial) and the other one (slots take turns)."""
    from visual_cortex_gb300 import synth
    from visual_cortex_gb300.batch import Batch, BatchError
    base = synth.make_workload("base", seed=43, nblock=4, n_lgn=512, m=20, width=64, height=64, nt=0, adex_inh=True,
                               nFrame=40, wFF=0.35, far_partners=60)
    trials = synth.batch_trials(n_trials=n, seed=43, base=base, width=64, height=64, nFrame=40, dur_ms=(5.0, 9.0))
    for limit in (0, 16, 512, 4096, -1):
        sims = [_sim(tr.wl) for tr in trials]
        try:
            for s in sims:
                native.check(s.plan, native.lib.pv1_set_wait_limit(s.plan, limit), "pv1_set_wait_limit")
            b = Batch(sims, [tr.steps for tr in trials], autotune=False)
            try:
                if limit == 0:
                    with pytest.raises(BatchError, match="device error word"):
                        b.sweep()
                else:
                    try:
                        b.sweep()
                    except BatchError as e:
                        assert limit > 0 and "device error word" in str(e)
            finally:
                b.close()
        finally:
            for s in sims:
                s.close()
