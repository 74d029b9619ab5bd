"""The surrogate-gradient adjoint at segment lengths, row lengths and sizes where its paths change, against
the unrolled PyTorch surrogate.

Tolerances as for the regular shapes: forward rates and mean potentials equal bit for bit (same
float32 operations in the same order), gradients to 2e-3 of the largest entry (another
summation order in the backward)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _patch(T, seg, win, bs=128, nE=96, nLGN=96, K=8, B=2, nblock=2, seed=0, rec_grad=False, cta_split=0, counts=1,
           density=0.2, drive=0.6):
    import torch
    from visual_cortex_gb300.adjoint import AdjointConfig, AdjointPatch
    rng = np.random.default_rng(seed)
    cfg = AdjointConfig(B=B, nblock=nblock, blockSize=bs, nE=nE, nLGN=nLGN, K=K, T=T, seg=seg, win=win,
                        rec_grad=rec_grad, cta_split=cta_split)
    ids = rng.integers(0, nLGN, size=(K, cfg.N)).astype(np.int32)
    X = (rng.random((B, T, nLGN)) < 0.01).astype(np.uint8) * rng.integers(1, counts + 1, (B, T, nLGN)).astype(np.uint8)
    nI = bs - nE
    Crec = (rng.random((nblock, nI, bs)) < density) * rng.uniform(0.05, 0.3, (nblock, nI, bs)) * min(1.0, 32.0 / nI)
    I0 = rng.uniform(0.0, drive, cfg.N).astype(np.float32)
    v0 = rng.uniform(-64.0, -52.0, (B, cfg.N)).astype(np.float32)
    patch = AdjointPatch(cfg, ids, X, Crec.astype(np.float32), I0, v0)
    return patch, torch.tensor(rng.uniform(0.1, 0.6, (K, cfg.N)), dtype=torch.float32, device="cuda")


def _gradients(patch, W, forward):
    import torch
    W = W.clone().requires_grad_(True)
    tE = torch.tensor(5.0, dtype=torch.float64, device="cuda", requires_grad=True)
    tI = torch.tensor(7.0, dtype=torch.float64, device="cuda", requires_grad=True)
    r, vb = forward(patch, W, tE, tI)
    target = torch.rand(r.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)) * 40
    (torch.mean((r - target) ** 2) + 0.1 * torch.mean((vb + 55.0) ** 2)).backward()
    return r.detach(), vb.detach(), W.grad, float(tE.grad), float(tI.grad)


def _check(patch, W):
    import torch
    from adjoint_reference import unrolled
    r, vb, g, e, i = _gradients(patch, W, lambda p, *a: p.forward(*a))
    r2, vb2, g2, e2, i2 = _gradients(patch, W, lambda p, W, tE, tI: unrolled(p, W, p.consts(tE, tI)))
    assert float(r2.sum()) > 0, "the test patch should spike"
    assert torch.equal(r, r2) and torch.equal(vb, vb2)
    assert float((g - g2).abs().max() / g2.abs().max()) < 2e-3
    assert abs(e - e2) <= 2e-3 * abs(e2) + 1e-8 and abs(i - i2) <= 2e-3 * abs(i2) + 1e-8


# last segments of 1, 55 and 2 steps, each followed by the segment before at a step of the same parity; and of 23
@pytest.mark.parametrize("cta_split", [1, 2])
@pytest.mark.parametrize("T,seg,win", [(65, 64, 65), (375, 64, 125), (200, 33, 100), (320, 99, 160)])
def test_last_segments(native, T, seg, win, cta_split):
    _check(*_patch(T, seg, win, seed=T, cta_split=cta_split))


@pytest.mark.parametrize("nLGN,counts,rec_grad", [(97, 1, False), (94, 3, True), (1100, 3, False), (60000, 2, False)])
def test_count_rows(native, nLGN, counts, rec_grad):
    """Rows of no whole words, of several words per thread, and with more cells than the event lists take."""
    _check(*_patch(130, 64, 65, nLGN=nLGN, counts=counts, rec_grad=rec_grad, seed=3))


@pytest.mark.parametrize("nE,density", [(512, 0.5), (768, 1.0), (992, 0.9)])
def test_room_for_inhibitory_weights(native, nE, density):
    """Blocks with more inhibitory neurons, more weights and not more than shared memory takes."""
    _check(*_patch(60, 16, 20, bs=1024, nE=nE, nblock=1, seed=nE, density=density, drive=2.0, cta_split=1))


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
def test_counts_at_any_address(native, offset):
    """Count rows are bytes: they may start anywhere."""
    import torch
    patch, W = _patch(130, 64, 65, seed=4)
    room = torch.zeros(patch.X.numel() + 4, dtype=torch.uint8, device="cuda")
    view = room[offset:offset + patch.X.numel()].view(patch.X.shape)
    view.copy_(patch.X)
    assert view.data_ptr() % 4 == offset % 4
    want = _gradients(patch, W, lambda p, *a: p.forward(*a))
    patch.X = view
    got = _gradients(patch, W, lambda p, *a: p.forward(*a))
    assert float(want[0].sum()) > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert float((got[2] - want[2]).abs().max() / want[2].abs().max()) < 1e-5


def test_two_threads_with_different_sizes(native):
    """Problems of different shared-memory sizes launched from two threads on their own streams."""
    import ctypes as C
    import threading
    import torch
    from visual_cortex_gb300.adjoint import AdjBuffers
    ptr = lambda t: C.c_void_p(t.data_ptr())
    calls, keep = [], []
    for q, kw in enumerate((dict(bs=512, nE=384, K=30, nLGN=4096), dict(bs=256, nE=192, K=16, nLGN=1024))):
        patch, W = _patch(1, 1, 1, B=1, nblock=1, seed=q, **kw)
        prob = patch._problem(patch.consts(torch.tensor(5.0), torch.tensor(7.0)))
        out = [torch.empty(patch.cfg.N, device="cuda") for _ in range(2)]
        ck = torch.empty(int(native.lib.pv1_adj_checkpoint_floats(C.byref(prob))), device="cuda")
        buf = AdjBuffers(ids=ptr(patch.ids), W=ptr(W), X=ptr(patch.X), Crec=ptr(patch.Crec), I0=ptr(patch.I0),
                         v0=ptr(patch.v0), rates=ptr(out[0]), vbar=ptr(out[1]), ck=ptr(ck))
        stream = torch.cuda.Stream()
        calls.append((prob, buf, C.c_void_p(stream.cuda_stream)))
        keep.append((patch, W, out, ck, stream))
    torch.cuda.synchronize()
    failed = [0, 0]

    def work(q):
        prob, buf, stream = calls[q]
        for _ in range(20000):
            failed[q] += native.lib.pv1_adj_forward(C.byref(prob), C.byref(buf), stream) != 0

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert failed == [0, 0]
