"""The work that is timed: what a program that uses the framework has it do.

Every case is one call sequence through the public entry points (Simulation, Batch,
AdjointPatch, LgnTensorCore) over the sizes of the synthetic configurations, from one block of
1,024 neurons stepped a few steps at a time to the full 32-block patch, the batched sweep, the
differentiable patch and the BF16 LGN stage.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from visual_cortex_gb300 import _native as N
from visual_cortex_gb300 import lgn_bf16, synth
from visual_cortex_gb300.adjoint import AdjointConfig, AdjointPatch, rate_loss
from visual_cortex_gb300.batch import Batch
from visual_cortex_gb300.model import FFLearning, Seeds, Simulation, Stimulus, host_init_state

f32 = np.float32
DT = 0.125          # ms, the step of every configuration
RATE_HZ = 15.0      # V1 rate of the synthetic patches, for the bytes and flops of work()


def listed():
    run = dict(kind="run", blockSize=1024, m=20, noise=False, far=0, movie=False)
    return [
        # closed-loop use: a small patch stepped 2 ms at a time, the raster read after each call;
        # launches, copies and waits count
        dict(run, name="patch1k_16steps", nblock=1, n_lgn=512, steps=16),
        # the smallest configuration in chunks of 100 ms (per-step latency on four CTAs)
        dict(run, name="patch1k_800steps", nblock=1, n_lgn=512, steps=800),
        # the patch size of the batched trials, alone, for an odd number of steps
        dict(run, name="patch8k_far_203steps", nblock=8, n_lgn=4096, steps=203, far=400),
        # the full patch end to end: the movie up, 100 ms of steps, the raster of every step down
        dict(run, name="patch32k_movie_800steps", nblock=32, n_lgn=16384, steps=800, far=400, movie=True),
        # membrane noise and synaptic failure on (the random-number paths of the step)
        dict(run, name="patch4k_noise_failure", nblock=4, n_lgn=2048, steps=301, noise=True),
        # the driver's output loop: raw state, LGN spikes and LGN rates of every step to the host
        dict(kind="record", name="record2k_96steps", nblock=2, blockSize=1024, n_lgn=512, m=20, far=100, steps=96),
        # LGN->V1 plasticity (triplet rule, homeostasis), weights read back after the chunk
        dict(kind="learn", name="learn2k_200steps", nblock=2, blockSize=1024, n_lgn=1024, m=20, far=0, steps=200),
        # a batched orientation sweep: trials of uneven length in one graph
        dict(kind="sweep", name="sweep12x4k", nblock=4, n_lgn=2048, m=20, far=400, trials=12, lo=400, hi=1600,
             chunked=False),
        # gradient of a small patch with the recurrent term, as a fitting loop on little data has it
        dict(kind="adjoint", name="adjoint_small", B=2, nblock=2, blockSize=128, nE=96, nLGN=96, K=8, T=320,
             rec_grad=True, vbar=True),
        # the differentiable patch: 4,096 neurons x 16 trials x 500 ms, forward and backward
        dict(kind="adjoint", name="adjoint_train", B=16, nblock=4, blockSize=1024, nE=768, nLGN=2048, K=30, T=4000,
             rec_grad=False, vbar=False),
        # the BF16 LGN stage on a short clip of few cells
        dict(kind="lgn", name="lgn_bf16_small", nCells=512, size=64, nFrame=24, side=15, T=640, fr_every=8),
        # the BF16 LGN stage at scale: 16,384 cells, 2 s of 256 x 256 noise
        dict(kind="lgn", name="lgn_bf16_full", nCells=16384, size=256, nFrame=240, side=31, T=16000, fr_every=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "record", "learn", "sweep", "adjoint", "lgn"])
    bs = rng.choice([1024, 1024, 768, 640, 512])
    if kind == "run":
        nb = _log(rng, 1, 24)
        noise = rng.random() < 0.2
        far = 0 if nb == 1 or noise else rng.choice([60, 200, 400])
        return dict(kind=kind, nblock=nb, blockSize=bs, n_lgn=512 * nb, m=rng.choice([12, 20, 24, 30]),
                    steps=_log(rng, 8, 800), noise=noise, far=far, movie=rng.random() < 0.3)
    if kind == "record":
        nb = rng.choice([1, 2, 3])
        return dict(kind=kind, nblock=nb, blockSize=bs, n_lgn=512 * nb, m=20, far=0 if nb == 1 else 100,
                    steps=rng.randrange(30, 200))
    if kind == "learn":
        nb = rng.choice([1, 2, 3, 4])
        return dict(kind=kind, nblock=nb, blockSize=bs, n_lgn=512 * nb, m=rng.choice([12, 20, 30]), far=0,
                    steps=rng.randrange(40, 300))
    if kind == "sweep":
        lo = rng.randrange(150, 500)
        return dict(kind=kind, nblock=rng.choice([1, 2, 4]), n_lgn=rng.choice([512, 1024, 2048]), m=20, far=200,
                    trials=rng.randrange(2, 11), lo=lo, hi=lo + rng.randrange(100, 1000), chunked=rng.random() < 0.3)
    if kind == "adjoint":
        bsz = rng.choice([128, 256, 512, 1024])
        return dict(kind=kind, B=_log(rng, 1, 16), nblock=rng.choice([1, 2, 3, 4]), blockSize=bsz, nE=bsz * 3 // 4,
                    nLGN=rng.choice([96, 250, 512, 1024, 2048]), K=rng.randrange(4, 33), T=160 * _log(rng, 1, 20),
                    rec_grad=rng.random() < 0.4, vbar=rng.random() < 0.5)
    side = rng.choice([15, 21, 31])
    return dict(kind=kind, nCells=_log(rng, 200, 12000), size=rng.choice([64, 96, 128]), nFrame=rng.randrange(24, 120),
                side=side, T=_log(rng, 500, 12000), fr_every=rng.choice([8, 16, 64]))


# ---- networks: drawn once per size, as a program reads its connectome files once ----

@functools.lru_cache(maxsize=None)
def _base(nblock, blockSize, n_lgn, m, far, noise):
    nE = blockSize * 3 // 4 if far == 0 else blockSize * 4 // 5
    size = 128 if nblock >= 8 else 64
    kw = dict(noisyDep=(0.2, 0.2), synFail=(0.1, 0.1, 0.1, 0.1), synFailFF=(0.1, 0.1)) if noise else {}
    return synth.make_workload("base", seed=7, nblock=nblock, blockSize=blockSize, nE=nE, n_lgn=n_lgn, m=m,
                               width=size, height=size, nt=0, far_partners=far, adex_inh=far > 0,
                               patch_deg=4.0 if nblock > 8 else 2.0, nFrame=240 if nblock > 8 else 120, **kw)


def _inputs(base, rng):
    """A drifting grating, an initial state and generator seeds of one trial."""
    lgn, fr = base.lgn, base.stim.frames
    xy = lgn.xy
    extent = 2 * (max(float(np.max(np.hypot(xy[:, 0], xy[:, 1]))), float(np.max(np.abs(xy)))) * 1.05 + 0.2)
    img = synth.grating_frames(fr.shape[0], fr.shape[3], fr.shape[2], extent, cpd=4.0, tf_hz=8.0,
                               contrast=float(rng.uniform(0.4, 1.0)), orient=float(rng.uniform(0, math.pi)),
                               frame_rate=120)
    spec, net = base.spec, base.net
    g = lambda row, n: np.tile(row, spec.nType * n).astype(f32)
    init = host_init_state(spec, int(rng.integers(1, 1 << 30)), net.tonicDep, net.nLGNperV1, None,
                           np.zeros(2 * spec.nType, f32), g([0.01, 0.2, 0.0, 0.2], spec.ngFF),
                           g([0.005, 0.2, 0.0, 0.2], spec.ngE), g([0.01, 0.2, 0.0, 0.2], spec.ngI))
    seeds = Seeds(lgn=int(rng.integers(1, 1 << 30)), cond=int(rng.integers(1, 1 << 30)),
                  trainDepth=base.seeds.trainDepth)
    return img, init, seeds


def _simulation(case, rng):
    base = _base(case["nblock"], case.get("blockSize", 1024), case["n_lgn"], case["m"], case["far"],
                 bool(case.get("noise")))
    img, init, seeds = _inputs(base, rng)
    frames = N.pinned_empty(img.shape, f32)
    frames[...] = img
    stim = Stimulus(frames=frames, init_LMS=(0.5, 0.5, 0.5))
    return Simulation(base.spec, base.net, base.lgn, stim, init, seeds), stim


# ---- the differentiable patch ----

def _adjoint_inputs(case, seed):
    rng = np.random.default_rng(seed)
    c = {k: case[k] for k in ("B", "nblock", "blockSize", "nE", "nLGN", "K", "T")}
    n, nI = c["nblock"] * c["blockSize"], c["blockSize"] - c["nE"]
    ids = rng.integers(0, c["nLGN"], size=(c["K"], n)).astype(np.int32)
    W = (rng.uniform(0.5, 1.5, size=(c["K"], n)) * (0.35 if c["K"] > 16 else 0.8)).astype(f32)
    # Poisson counts of LGN cells whose rate is modulated at 8 Hz, each cell at its own phase
    t = np.arange(c["T"])[:, None] * DT * 1e-3
    phase = rng.uniform(0, 2 * np.pi, c["nLGN"])[None, :]
    p = ((25 + 20 * np.sin(2 * np.pi * 8 * t + phase)) * DT * 1e-3).astype(f32)
    X = np.empty((c["B"], c["T"], c["nLGN"]), np.uint8)
    for b in range(c["B"]):
        u = rng.random(p.shape, dtype=f32)
        X[b] = (u < p).astype(np.uint8) + (u < 0.02 * p).astype(np.uint8)
    Crec = np.where(rng.random((c["nblock"], nI, c["blockSize"]), dtype=f32) < 0.2,
                    0.25 * rng.lognormal(0.0, 0.5, (c["nblock"], nI, c["blockSize"])), 0).astype(f32)
    I0 = rng.uniform(0.0, 0.3, n).astype(f32)
    v0 = rng.uniform(-65.0, -55.0, (c["B"], n)).astype(f32)
    target = rng.uniform(0.0, 40.0, (c["B"], c["T"] // 160, n)).astype(f32)
    return c, ids, W, X, Crec, I0, v0, target


def _loss(rates, vbar, target, case):
    loss = rate_loss(rates, target)
    return loss + 0.1 * torch.mean((vbar + 58.0) ** 2) if case["vbar"] else loss


# ---- the BF16 LGN stage ----

@functools.lru_cache(maxsize=None)
def _lgn_base(nCells, size, nFrame, side, T):
    return lgn_bf16.make_workload(nCells=nCells, size=size, nFrame=nFrame, side=side, T=T, seed=3)


def _lgn_workload(case, seed):
    """The stage's cells and frame weights with a movie of 1/f^2 noise drawn from the seed."""
    base = _lgn_base(*(case[k] for k in ("nCells", "size", "nFrame", "side", "T")))
    n, size = case["nFrame"], case["size"]
    gen = torch.Generator().manual_seed(seed)
    fx = torch.fft.fftfreq(size)
    f = torch.hypot(fx[:, None], fx[None, :])
    f[0, 0] = 1.0
    amp = 1.0 / f
    amp[0, 0] = 0.0
    w = torch.randn(n, size, size, generator=gen).cuda()
    x = torch.fft.ifft2(torch.fft.fft2(w) * amp.cuda()).real
    x = (x - x.mean((1, 2), keepdim=True)) / x.std((1, 2), keepdim=True)
    frames = torch.clamp(0.5 * (1 + 0.3 * x), 0.0, 1.0).float().cpu().numpy()
    return dataclasses.replace(base, frames=frames)


class _DeviceArray:
    """A device array of the framework as torch sees it (no copy); the tensor has to keep
    the array's owner alive."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f4", data=(int(ptr), False), version=3)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("run", "record", "learn"):
        sim, stim = _simulation(case, rng)
        s = dict(case=case, sim=sim, stim=stim)
        if kind == "record":
            sim.set_record(N.REC_RAW | N.REC_LGN_SP | N.REC_LGN_FR, case["steps"] + 1)
            return s
        if kind == "learn":
            sim.set_ff_learning(FFLearning(
                tauLTP=16.8, tauLTD=33.7, tauTrip=114.0, tauAvg=1000.0, targetFR=0.0, A_LGN=0.02, r_LTD=1.0,
                gmaxLGN=0.6, gminLGN=0.0, sRatioLGN=1.0, decayTimeHomeoFF=250.0, FF_InfRatio=1.0, applyHomeo=1))
        sim.set_record(N.REC_SPIKES, case["steps"] + 1)
        s["raster"] = N.pinned_empty((case["steps"], sim.spec.nV1), f32)
        return s
    if kind == "sweep":
        sims = [_simulation(case, rng)[0] for _ in range(case["trials"])]
        steps = [int(x) for x in rng.integers(case["lo"], case["hi"] + 1, case["trials"])]
        # every seed has the same longest trial, so that passes of different seeds compare
        steps[0], steps[-1] = case["hi"], case["lo"]
        return dict(case=case, sims=sims, steps=steps)
    if kind == "adjoint":
        c, ids, W, X, Crec, I0, v0, target = _adjoint_inputs(case, seed)
        patch = AdjointPatch(AdjointConfig(rec_grad=case["rec_grad"], **c), ids, X, Crec, I0, v0)
        return dict(case=case, patch=patch, W=torch.from_numpy(W).cuda(), target=torch.from_numpy(target).cuda(),
                    tau=torch.tensor([5.0, 7.0]).cuda())
    wl = _lgn_workload(case, seed)
    return dict(case=case, tc=lgn_bf16.LgnTensorCore(wl, fr_every=case["fr_every"]), seed=seed)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        if case["movie"]:
            state["sim"].load_stimulus(state["stim"])
        return dict(raster=state["sim"].run_spikes_to_host(case["steps"], state["raster"]))
    if kind == "record":
        sim, k = state["sim"], case["steps"]
        first = sim.step
        sim.run(k)
        raw, sp, fr = sim.fetch_records(first, k, raw=True, lgn_sp=True, lgn_fr=True)
        return dict(raw=raw, lgn_sp=sp, lgn_fr=fr)
    if kind == "learn":
        raster = state["sim"].run_spikes_to_host(case["steps"], state["raster"])
        return dict(raster=raster, sLGN=state["sim"].state("sLGN"))
    if kind == "sweep":
        b = Batch(state["sims"], state["steps"], autotune=False)
        if case["chunked"]:
            b.run()
        else:
            b.sweep()
        rates = [b.stats(q, rates=True)[2] for q in range(len(state["sims"]))]
        b.close()
        return dict(rates=np.concatenate(rates), v=np.concatenate([s.state("v") for s in state["sims"]]))
    if kind == "adjoint":
        W = state["W"].detach().requires_grad_(True)
        tau = state["tau"].detach().requires_grad_(True)
        rates, vbar = state["patch"].forward(W, tau[0], tau[1])
        _loss(rates, vbar, state["target"], case).backward()
        return dict(rates=rates.detach(), vbar=vbar.detach(), gW=W.grad, gTau=tau.grad)
    tc = state["tc"]
    tc.run(tensor_cores=True, seed=state["seed"])
    rates = tc.fetch()[2]
    spikes = torch.as_tensor(_DeviceArray(tc.device_spikes(), (case["T"], case["nCells"])), device="cuda")
    spikes.owner = tc
    return dict(rates=rates, spikes=spikes)


def work(case):
    kind = case["kind"]
    if kind == "adjoint":
        n = case["B"] * case["nblock"] * case["blockSize"]
        per = case["nblock"] * case["blockSize"]
        nI = case["blockSize"] - case["nE"]
        win = case["T"] // 160
        b = case["B"] * case["T"] * case["nLGN"] + 4 * (3 * case["K"] * per + per + n + 4 * n * win) + 4 * nI * per
        # forward, recompute and adjoint: about 45 + 45 + 80 operations per neuron-step
        return dict(bytes=b, flops=170.0 * n * case["T"] + 6.0 * 0.004 * case["K"] * n * case["T"])
    if kind == "lgn":
        cells, T = case["nCells"], case["T"]
        # the bf16 spatial table and the frame weights in, spike words and recorded rates out
        b = 2 * cells * case["nFrame"] + 128 * T + 4 * T * cells + 4 * (T // case["fr_every"]) * cells
        return dict(bytes=b, flops=(2.0 * 32 + 20) * T * cells)
    nb, bs = case["nblock"], case.get("blockSize", 1024)
    n = nb * bs
    S = 3 + 2 * (2 + 2 + 1)
    if kind == "sweep":
        copies, steps = case["trials"], (case["lo"] + case["hi"]) / 2
        out = copies * n * 12
    else:
        copies, steps = 1, case["steps"]
        out = 4 * n * steps if kind != "record" else 4 * steps * (n * (S + 2) + 2 * case["n_lgn"])
        if kind == "learn":
            out += 8 * case["m"] * n
    ns = copies * n * steps
    spikes = RATE_HZ * DT * 1e-3 * ns
    events = spikes * (case["far"] + bs / 10)
    b = copies * n * (8 * S + 8 * case["m"]) + out + spikes * 4 * bs + spikes * case["far"] * 16
    if case.get("movie"):
        side = 128 if nb >= 8 else 64
        b += 3 * 4 * side * side * (240 if nb > 8 else 120)
    # membrane step about 150 operations, an event about 20; LGN: 32 frames and the rate per cell-step
    return dict(bytes=b, flops=150.0 * ns + 20.0 * events + 90.0 * copies * case["n_lgn"] * steps)


# ---- 64-bit values of the computed outputs ----

def _exact_adjoint(case, seed):
    """The patch unrolled step by step in float64 on torch, gradients by autograd."""
    c, ids, W, X, Crec, I0, v0, target = _adjoint_inputs(case, seed)
    if case["B"] * case["nblock"] * case["blockSize"] * case["T"] * case["K"] > 2e8:
        return None
    d = lambda a: torch.from_numpy(a).cuda().double()
    B, T, bs, nE = c["B"], c["T"], c["blockSize"], c["nE"]
    W, tau, I0, Crec, target = d(W).requires_grad_(True), torch.tensor([5.0, 7.0]).cuda().double(), d(I0), d(Crec), d(target)
    tau.requires_grad_(True)
    X, ids = torch.from_numpy(X).cuda(), torch.from_numpy(ids).cuda().long()
    n = I0.numel()

    class Spike(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            ctx.save_for_backward(x)
            return (x > 0).double()

        @staticmethod
        def backward(ctx, g):
            (x,) = ctx.saved_tensors
            return g / (1 + 5.0 * x.abs()) ** 2

    decay = [torch.exp(-DT / t) for t in tau]
    rise = math.exp(-DT / 1.0)
    dod = [1.0 / (t - 1.0) for t in tau]
    isE = (torch.arange(n, device="cuda") % bs) < nE
    tRef = torch.where(isE, 16, 8)
    v = d(v0)
    gE = hE = gI = hI = torch.zeros(B, n, device="cuda", dtype=torch.float64)
    ref = torch.zeros(B, n, device="cuda", dtype=torch.long)
    rates, vbar, cnt, vs = [], [], 0.0, 0.0
    for t in range(T):
        gE1 = gE * decay[0] + hE * dod[0] * (decay[0] - rise)
        gI1 = gI * decay[1] + hI * dod[1] * (decay[1] - rise)
        hE1, hI1 = hE * rise, hI * rise
        dv = lambda u, e, i: -0.05 * (u + 65.0) - e * u - i * (u + 75.0) + I0
        k1 = dv(v, gE, gI)
        k2 = dv(v + DT * k1, gE1, gI1)
        vn = v + 0.5 * DT * (k1 + k2)
        free = ref == 0
        fired = free & (vn > -50.0)
        s = torch.where(free, Spike.apply(vn + 50.0), torch.zeros_like(vn))
        v = torch.where(free & ~fired, vn, torch.full_like(vn, -60.0))
        ref = torch.where(fired, tRef, (ref - 1).clamp(min=0))
        hE = hE1 + (W * X[:, t][:, ids].double()).sum(1)
        sI = (s if case["rec_grad"] else s.detach()).view(B, -1, bs)[:, :, nE:]
        hI = hI1 + torch.einsum("bki,kij->bkj", sI, Crec).reshape(B, n)
        gE, gI = gE1, gI1
        cnt, vs = cnt + s, vs + v
        if (t + 1) % 160 == 0:
            rates.append(cnt / (160 * DT * 1e-3))
            vbar.append(vs / 160)
            cnt, vs = 0.0, 0.0
    rates, vbar = torch.stack(rates, 1), torch.stack(vbar, 1)
    loss = torch.mean((rates - target) ** 2)
    if case["vbar"]:
        loss = loss + 0.1 * torch.mean((vbar + 58.0) ** 2)
    loss.backward()
    return dict(rates=rates.detach(), vbar=vbar.detach(), gW=W.grad, gTau=tau.grad)


def _exact_lgn(case, seed):
    """The rates at the recorded steps: contrast sums, frame weights and logistic in float64."""
    wl = _lgn_workload(case, seed)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().double()
    size, side, n = case["size"], wl.side, case["nCells"]
    half = side // 2
    q = torch.arange(side * side, device="cuda")
    x = torch.from_numpy(wl.cx).cuda().long()[:, None] + q % side - half
    y = torch.from_numpy(wl.cy).cuda().long()[:, None] + q // side - half
    inside = (x >= 0) & (x < size) & (y >= 0) & (y < size)
    at = torch.where(inside, y * size + x, 0)
    sw = d(wl.SW) * inside
    S = torch.zeros(n, wl.nFext, device="cuda", dtype=torch.float64)
    frames = d(wl.frames).reshape(case["nFrame"], -1)
    for col in range(lgn_bf16.PAD, wl.nFext):
        c = torch.clamp(frames[(col - lgn_bf16.PAD) % case["nFrame"]] / wl.meanLum - 1, -1, 1)
        S[:, col] = (sw * c[at]).sum(1)
    S = torch.nn.functional.pad(S, (0, lgn_bf16.TILE_K))
    steps = np.arange(0, case["T"], case["fr_every"])
    W = d(wl.W)
    out = torch.empty(len(steps), n, device="cuda", dtype=torch.float64)
    k, mx, c50, sharp, la, lb = (d(a) for a in (np.abs(wl.k), wl.maxConvol, wl.c50, wl.sharp, wl.la, wl.lb))
    for i, t in enumerate(steps):
        tile, f0 = int(t) // lgn_bf16.TILE_N, int(wl.f0[int(t) // lgn_bf16.TILE_N])
        conv = S[:, f0:f0 + lgn_bf16.TILE_K] @ W[tile, int(t) % lgn_bf16.TILE_N]
        current = torch.clamp(conv * k * wl.convolRatio, min=0.0)
        out[i] = wl.frRatio * mx * (la / (1 + torch.exp(sharp * (c50 - current / mx))) + lb)
    return dict(rates=out.cpu().numpy(), spikes=None)


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] == "lgn":
        return _exact_lgn(case, seed)
    return None   # spiking networks on drawn random numbers: no value but the run's own
