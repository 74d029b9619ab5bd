"""Generator seeding: every cell's MRG32k3a state sits 2^76 draws after the one before it.

The states are compared word for word with the recurrence's jump matrices A^(2^76 * id), built
here from the published recurrence by repeated squaring in Python integers, over sequence
numbers past 2^16 (every bit count and carry of the device's per-bit products)."""
import numpy as np
import pytest

M = (2**32 - 209, 2**32 - 22853)
A = ([[0, 1, 0], [0, 0, 1], [-810728, 1403580, 0]], [[0, 1, 0], [0, 0, 1], [-1370589, 0, 527612]])


def _square(a, m):
    return [[sum(a[i][k] * a[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]


def _sequences(first, n, m, a):
    """States of sequences 0..n-1 from that of sequence 0, by doubling."""
    for _ in range(76):
        a = _square(a, m)
    out = np.array([first], np.uint64)
    while len(out) < n:
        J = np.array([[x % m for x in row] for row in a], np.uint64)
        prod = (out[:, None, :] * J[None, :, :]) % np.uint64(m)
        out = np.concatenate([out, prod.sum(2, dtype=np.uint64) % np.uint64(m)])
        a = _square(a, m)
    return out[:n]


def test_sequences_commute_with_draws():
    """CPU: one draw after the jump equals the jump after one draw (the doubling above is a power of A)."""
    for m, a in zip(M, A):
        x = np.array([[123456789, 362436069, 521288629]], np.uint64)
        step = np.array([[v % m for v in row] for row in a], np.uint64)
        draw = lambda s: ((s[:, None, :] * step[None]) % np.uint64(m)).sum(2, dtype=np.uint64) % np.uint64(m)
        s = _sequences(x[0], 9, m, a)
        np.testing.assert_array_equal(draw(s), _sequences(draw(x)[0], 9, m, a))


@pytest.mark.gpu
@pytest.mark.parametrize("n_lgn,seed", [(70001, 3), (514, 2**31 + 11)])
def test_states_are_jumps_of_the_first(native, n_lgn, seed):
    from visual_cortex_gb300 import synth
    from visual_cortex_gb300.model import Seeds, Simulation
    wl = synth.make_workload("rng", seed=1, nblock=1, blockSize=640, nE=512, n_lgn=n_lgn, m=8, width=32, height=32,
                             nt=8, nFrame=4, mSample1D=8)
    sim = Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, Seeds(lgn=seed, cond=seed + 5, trainDepth=3))
    try:
        lgn = sim.state("lgn_rng").reshape(-1, 48)
        cond, noisy = (sim.state(k).reshape(-1, 48) for k in ("v1_rng_cond", "v1_rng_noisy"))
    finally:
        sim.close()
    words = lambda s: np.ascontiguousarray(s[:, :24]).view(np.uint32).astype(np.uint64)
    for s in (lgn, cond):
        for q, (m, a) in enumerate(zip(M, A)):
            w = words(s)[:, 3 * q:3 * q + 3]
            np.testing.assert_array_equal(w, _sequences(w[0], len(w), m, a))
    # rNoisy starts nV1 sequences further on and has drawn nothing: trainDepth draws bring it to
    # where rGenCond's continuation would be
    n = wl.spec.nV1
    for q, (m, a) in enumerate(zip(M, A)):
        step = np.array([[v % m for v in row] for row in a], np.uint64)
        w = words(noisy)[:, 3 * q:3 * q + 3]
        for _ in range(3):
            w = ((w[:, None, :] * step[None]) % np.uint64(m)).sum(2, dtype=np.uint64) % np.uint64(m)
        np.testing.assert_array_equal(w, _sequences(words(cond)[0, 3 * q:3 * q + 3], 2 * n, m, a)[n:])
    assert not lgn[:, 24:].any()
