"""Far events left by one V1 kernel for the next: the per-step kernel leaves a step's list of far spikers,
which whichever kernel runs the following step pushes, once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("v", "w", "tBack", "gE", "hE", "gI", "hI", "gFF", "hFF")


def _sim(wl):
    from visual_cortex_gb300.model import Simulation
    return Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)


def test_tuned_batch_of_more_trials_than_slots(native):
    """30 trials of 12 CTAs each, more than are resident at once, so that a slot's CTAs come to its next trial at
    different times.  The tuning alternates per-step and persistent chunks (24 of them within 900 steps):
    every trial ends as it does alone."""
    from visual_cortex_gb300 import synth
    from visual_cortex_gb300.batch import Batch
    base = synth.make_workload("handover", seed=5, nblock=6, blockSize=512, nE=384, n_lgn=512, m=20, width=64, height=64,
                               nt=0, nFrame=60, far_partners=120, adex_inh=True, wFF=0.35, wFar=0.01)
    trials = synth.batch_trials(n_trials=30, seed=5, base=base, width=64, height=64, nFrame=60, dur_ms=(114.0, 125.0))
    batched = [_sim(tr.wl) for tr in trials]
    try:
        b = Batch(batched, [tr.steps for tr in trials], autotune=True)
        try:
            assert b.run()[0] == 0
            assert min(b.tuning()["ms_per_chunk"].values()) > 0     # every variant ran
            assert min(b.stats(q)[1] for q in range(len(trials))) > 1.0
        finally:
            b.close()
        for q, tr in enumerate(trials):
            alone = _sim(tr.wl)
            try:
                alone.persistent(0)
                alone.run(tr.steps)
                for k in STATE:
                    np.testing.assert_array_equal(batched[q].state(k), alone.state(k), err_msg=f"trial {q} {k}")
            finally:
                alone.close()
    finally:
        for s in batched:
            s.close()
