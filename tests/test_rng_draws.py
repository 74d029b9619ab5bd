"""The uniforms of the LGN's Poisson generators, draw for draw: the published recurrence of MRG32k3a in Python integers,
its output over m1 rounded to float, from each cell's state at the start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M1, M2 = 2**32 - 209, 2**32 - 22853


def _draws(s, n):
    a, b = [int(x) for x in s[:3]], [int(x) for x in s[3:6]]
    out = np.empty(n, np.float32)
    for k in range(n):
        p1 = (1403580 * a[1] - 810728 * a[0]) % M1
        p2 = (527612 * b[2] - 1370589 * b[0]) % M2
        a, b = [a[1], a[2], p1], [b[1], b[2], p2]
        z = p1 - p2 if p1 > p2 else p1 - p2 + M1
        out[k] = np.float32(float(z) * (1.0 / 4294967087.0))
    return out


@pytest.mark.parametrize("n_parvo", [0, 64])
def test_uniforms_are_the_published_recurrence(native, n_parvo):
    from visual_cortex_gb300 import synth
    from visual_cortex_gb300.model import Simulation
    kw = dict(n_parvo=n_parvo, tau=300.0, nKernelSample=150) if n_parvo else {}
    wl = synth.make_workload("draws", seed=61, nblock=1, blockSize=256, nE=192, n_lgn=256, m=20, width=64, height=64,
                             nt=800, nFrame=60, **kw)
    sim = Simulation(wl.spec, wl.net, wl.lgn, wl.stim, wl.init, wl.seeds)
    try:
        state = np.ascontiguousarray(sim.state("lgn_rng").reshape(-1, 48)[:, :24]).view(np.uint32)
        sim.set_draw_record(800, 6)
        sim.run(800)
        u, counts = sim.fetch_draws(0)
    finally:
        sim.close()
    u, counts = u.reshape(800, len(state), 6), counts.reshape(800, len(state))
    assert counts.sum() > 200 and counts.max() <= 6
    for c in range(len(state)):
        got = np.concatenate([u[t, c, :counts[t, c]] for t in np.flatnonzero(counts[:, c])] or [np.empty(0, np.float32)])
        np.testing.assert_array_equal(got, _draws(state[c], len(got)), err_msg=f"cell {c}")
