// Surrogate-gradient adjoint of a conductance-based LIF patch (the differentiable form).
//
// The reference has no gradient code; this is the differentiable counterpart of its V1 step
// (src/coredynamics.cu:1235-2059 with the two-state conductance kernel of
// src/condShape.h:13-51), on batches of trials:
//   conductances  g' = g*Ed + h*dod*(Ed - Er),  h' = h*Er   (Ed = e^{-dt/td}, Er = e^{-dt/tr},
//                 dod = tr/(td - tr)), AMPA from the LGN, GABA from the block's I neurons;
//   membrane      RK2 (Heun) of dv/dt = -gL(v-vL) - gE(v-vE) - gI(v-vI) + I0 with the
//                 conductances of the start and of the end of the step, as the reference;
//   spikes        s = H(vn - vThres) forward, ds/dvn = 1/(1 + slope|vn - vThres|)^2 (fast
//                 sigmoid) backward; reset to vR with the reset gate held constant; refractory
//                 steps hold v at vR;
//   inputs        end of step t: hE += sum_k W[k][n] X[t][id[k][n]] (k ascending),
//                 hI += sum of C[p][n] over the I neurons p of the block that spiked (ascending);
//   outputs       per window of `win` steps: spike rate (Hz) and mean membrane potential.
// Spikes are delivered at step granularity (no sub-step spike-time offsets).
//
// One CTA (or a cluster of ctaSplit CTAs sharing the block's spike ballots and adjoints through
// distributed shared memory) holds one (trial, block) pair, one thread per neuron; blocks do
// not interact.  The
// forward stores a checkpoint of (v, gE, hE, gI, hI, refractory count) every `seg` steps; the
// backward walks the segments from the last one, recomputes each forward from its checkpoint
// into a per-CTA scratch, then runs the adjoint backwards through it.  The recurrent term of
// the adjoint (sum over posts of C[p][n] * lambda_hI[n] for every I neuron p) is a
// warp-cooperative mat-vec over the block's C rows per step.  Gradients: dL/dW by atomic adds
// at the (sparse) LGN events, dL/d(EdE, ErE, dodE, EdI, ErI, dodI) reduced in FP64.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include <cooperative_groups.h>

#include "pv1_internal.cuh"

namespace cg = cooperative_groups;

namespace {

thread_local std::string g_adjErr;

struct AdjArgs {
    pv1_adj_problem p;
    pv1_adj_buffers b;
    int N, nI, nWin, nSeg;
    int split;   // CTAs per (trial, block)
    // dynamic shared memory, in bytes from its start (-1: not there): event masks of the CTA's neurons,
    // their event lists by LGN cell (offsets, entries), synapse weights, inhibitory weights
    int maskAt, offAt, entAt, wAt;
    int gabaAt, gabaRoom;   // the block's inhibitory weights
    int smemBytes;
};

// Exchange between the CTAs of a (trial, block): a block of one CTA stores to its own shared memory;
// with two, floats go to both through the cluster's distributed shared memory.
__device__ __forceinline__ void share_float(float *addr, float v, int split) {
    if (split == 1) {
        *addr = v;
        return;
    }
    cg::cluster_group cl = cg::this_cluster();
    for (int r = 0; r < split; r++) *cl.map_shared_rank(addr, r) = v;
}

__device__ __forceinline__ void store_at_rank(float *addr, float v, int rank, int split) {
    if (split == 1) {
        *addr = v;
        return;
    }
    *cg::this_cluster().map_shared_rank(addr, rank) = v;
}

// Barrier over the (trial, block)'s CTAs (with the memory ordering of their shared writes).
__device__ __forceinline__ void block_sync(int split) {
    if (split == 1) __syncthreads();
    else cg::this_cluster().sync();
}

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

constexpr int kAdjMaxK = 32;

struct AState {
    float v, gE, hE, gI, hI;
    int ref;
};

__device__ __forceinline__ float adj_f(float v, float gE, float gI, float gL, float vL, float vE, float vI,
                                       float I0) {
    return -gL * (v - vL) - gE * (v - vE) - gI * (v - vI) + I0;
}

// Forward step of one neuron up to the spike decision; returns v_next, sets spk, refr and the
// decayed conductances.  Shared by the forward and the recompute of the backward.
__device__ __forceinline__ float adj_neuron_step(const pv1_adj_problem &P, AState &s, float I0, bool isE,
                                                 bool &spk, bool &refr, float &gE1, float &hE1, float &gI1,
                                                 float &hI1) {
    gE1 = s.gE * P.EdE + s.hE * P.dodE * (P.EdE - P.ErE);
    hE1 = s.hE * P.ErE;
    gI1 = s.gI * P.EdI + s.hI * P.dodI * (P.EdI - P.ErI);
    hI1 = s.hI * P.ErI;
    refr = s.ref > 0;
    spk = false;
    if (refr) {
        s.ref -= 1;
        return P.vR;
    }
    const float k1 = adj_f(s.v, s.gE, s.gI, P.gL, P.vL, P.vE, P.vI, I0);
    const float v1 = s.v + P.dt * k1;
    const float k2 = adj_f(v1, gE1, gI1, P.gL, P.vL, P.vE, P.vI, I0);
    const float vn = s.v + (P.dt * 0.5f) * (k1 + k2);
    spk = vn > P.vThres;
    if (spk) {
        s.ref = (int)(isE ? P.tRefE : P.tRefI);
        return P.vR;
    }
    return vn;
}

// ---- what a step hands over inside a (trial, block) ----
// Two things cross threads in a step: the spikes of the block's inhibitory neurons, and the LGN
// events.  Polling every neuron's K synapses (K byte gathers and K id loads per neuron-step) was
// most of the step, while in a step only a fraction of a percent of the cells spike.  So each
// CTA keeps, per LGN cell, the list of its (neuron, synapse) pairs; the threads scan the step's
// count row together and set, for the few cells with events, the synapse's bit in the neuron's
// mask.  A neuron then visits its set bits in ascending synapse order, so that its sums are those
// of the full walk.  The warps' ballots go to every CTA of the block as asynchronous stores that
// count towards an mbarrier; the same mbarrier tells that every warp has set its bits.  Two
// buffers by parity of a running count of exchanges: a warp reaches exchange e + 2's only after the
// phase of exchange e + 1, which its peers announce after they have used exchange e's.  (Not by parity
// of the step: the backward goes from the last step to the segment before, which can have the
// same one.)
// Measured, with the staged inhibitory weights below: forward and backward of 4,096 neurons x 16 trials x
// 4,000 steps 40,384 -> 22,530 us (some 1,600 more without them), of two blocks of 128 neurons x 320 steps
// with the recurrent term 3,784 -> 2,914 us (1,737 with one CTA per block, as adj_check chooses now).
struct AdjShared {
    unsigned ball[2][32];
    unsigned *mask[2], *many[2];   // per neuron of the CTA: synapses with an event; those with a count above 1
    uint64_t bar[2];
    int scan[32];
};

// Entry of an event list: neuron of the CTA (10 bits), synapse (5 bits).
__device__ __forceinline__ void build_events(const AdjArgs &A, uint8_t *dyn, int firstN, int nNeurons, AdjShared &sm) {
    if (A.entAt < 0) return;
    unsigned *off = reinterpret_cast<unsigned *>(dyn + A.offAt);   // [nLGN + 1]
    unsigned short *ent = reinterpret_cast<unsigned short *>(dyn + A.entAt);
    const int L = (int)A.p.nLGN, K = (int)A.p.K;
    for (int c = threadIdx.x; c <= L; c += blockDim.x) off[c] = 0u;
    __syncthreads();
    for (int q = threadIdx.x; q < K * nNeurons; q += blockDim.x) {
        const int k = q / nNeurons, j = q - k * nNeurons;
        atomicAdd(&off[__ldg(A.b.ids + (size_t)k * A.N + firstN + j)], 1u);
    }
    __syncthreads();
    // exclusive scan: each thread a run of cells, the runs' totals by one warp
    const int T = blockDim.x, per = (L + T - 1) / T;
    const int c0 = min(L, (int)threadIdx.x * per), c1 = min(L, c0 + per);
    unsigned sum = 0;
    for (int c = c0; c < c1; c++) sum += off[c];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) sm.scan[warp] = (int)incl;
    __syncthreads();
    unsigned run = incl - sum;
    for (int w = 0; w < warp; w++) run += (unsigned)sm.scan[w];
    for (int c = c0; c < c1; c++) {
        const unsigned n = off[c];
        off[c] = run;
        run += n;
    }
    __syncthreads();
    // off[c] runs to the end of its list while the entries are placed: afterwards list c is
    // [off[c - 1], off[c])
    for (int q = threadIdx.x; q < K * nNeurons; q += blockDim.x) {
        const int k = q / nNeurons, j = q - k * nNeurons;
        const unsigned at = atomicAdd(&off[__ldg(A.b.ids + (size_t)k * A.N + firstN + j)], 1u);
        ent[at] = (unsigned short)(j << 5 | k);
    }
    __syncthreads();
}

// One cell's events of a step into the masks of the CTA's neurons.
__device__ __forceinline__ void mark_cell(const unsigned *off, const unsigned short *ent, int cell, unsigned count,
                                          unsigned *mask, unsigned *many) {
    const unsigned e1 = off[cell];
    for (unsigned e = cell ? off[cell - 1] : 0u; e < e1; e++) {
        const unsigned v = ent[e];
        atomicOr(&mask[v >> 5], 1u << (v & 31));
        if (count > 1) atomicOr(&many[v >> 5], 1u << (v & 31));
    }
}

// A thread's share of a count row, fetched a step ahead: up to two words of four cells each (aligned rows of
// whole words with no more than eight cells per thread), else nothing (the row is read when marked).
struct RowShare {
    unsigned w[2];
};

__device__ __forceinline__ bool row_fits(const AdjArgs &A) {
    return A.entAt >= 0 && A.p.nLGN % 4 == 0 && A.p.nLGN <= 8 * blockDim.x &&
           reinterpret_cast<uintptr_t>(A.b.X) % 4 == 0;
}

__device__ __forceinline__ RowShare fetch_row(const AdjArgs &A, const uint8_t *row, bool fits) {
    RowShare r{{0u, 0u}};
    if (fits) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const unsigned c = (threadIdx.x + k * blockDim.x) * 4;
            if (c < A.p.nLGN) r.w[k] = __ldg(reinterpret_cast<const unsigned *>(row + c));
        }
    }
    return r;
}

// The events of a count row into the masks of exchange parity par: each thread its share of the cells.
__device__ __forceinline__ void mark_events(const AdjArgs &A, const uint8_t *dyn, const uint8_t *row, const RowShare &r,
                                            bool fits, AdjShared &sm, int par) {
    if (A.entAt < 0) return;
    const unsigned *off = reinterpret_cast<const unsigned *>(dyn + A.offAt);
    const unsigned short *ent = reinterpret_cast<const unsigned short *>(dyn + A.entAt);
    if (fits) {
#pragma unroll
        for (int k = 0; k < 2; k++) {
            unsigned w = r.w[k];
            while (w) {
                const int byte = (__ffs(w) - 1) >> 3;
                const unsigned count = (w >> (8 * byte)) & 0xffu;
                w &= ~(0xffu << (8 * byte));
                mark_cell(off, ent, (threadIdx.x + k * blockDim.x) * 4 + byte, count, sm.mask[par], sm.many[par]);
            }
        }
    } else {
        for (int c = threadIdx.x; c < (int)A.p.nLGN; c += blockDim.x) {
            const unsigned count = __ldg(row + c);
            if (count) mark_cell(off, ent, c, count, sm.mask[par], sm.many[par]);
        }
    }
}

// Announces this warp's part of an exchange (its bits are set, its ballot is on the way) to every CTA of the
// block.
__device__ __forceinline__ void send_ballot(AdjShared &sm, int par, int word, unsigned bal, int split) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const unsigned bar = smem_u32(&sm.bar[par]);
    if (split == 1) {
        if (lane == 0) {
            sm.ball[par][word] = bal;
            asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
        }
        return;
    }
    if (lane < split) {
        unsigned addr, peer;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&sm.ball[par][word])), "r"(lane));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(bar), "r"(lane));
        asm volatile("fence.acq_rel.cta;" ::: "memory");   // the bits set in this CTA's masks
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(bal),
                     "r"(peer)
                     : "memory");
        asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], 4;" ::"r"(peer) : "memory");
    }
}

// Bounded wait of a warp for the phase of an exchange's parity; false if it does not complete.  A poll suspends
// the warp for up to 3.9 us: the limit is a second.
constexpr int kAdjSpins = 1 << 18;
__device__ __forceinline__ bool wait_block(AdjShared &sm, int par, unsigned &phase) {
    const unsigned bar = smem_u32(&sm.bar[par]);
    const unsigned want = (phase >> par) & 1u;
    unsigned ok = 0u;
    for (int i = 0; i < kAdjSpins && !ok; i++)
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(bar), "r"(want)
            : "memory");
    if (!__all_sync(0xffffffffu, ok)) return false;
    phase ^= 1u << par;
    return true;
}

// The neuron's LGN events of a step into hE, synapse order; returns their mask.  Without event lists
// (they did not fit) every synapse's count is read.  ids: the global array (stride N); weights: a
// shared-memory copy (stride blockDim.x) or the global array.
struct SynView {
    const int32_t *ids;
    const float *W;
    int wStride;
};

__device__ __forceinline__ unsigned lgn_inputs(const AdjArgs &A, const uint8_t *x, AdjShared &sm, int par, float &hE,
                                               SynView sv, bool &many) {
    unsigned mask;
    if (A.entAt >= 0) {
        mask = sm.mask[par][threadIdx.x];
        unsigned more = 0u;
        if (mask) {
            more = sm.many[par][threadIdx.x];
            sm.mask[par][threadIdx.x] = 0u;
            if (more) sm.many[par][threadIdx.x] = 0u;
        }
        many = more != 0u;
        for (unsigned m = mask; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            const float c = (more >> k) & 1u ? (float)__ldg(x + __ldg(sv.ids + (size_t)k * A.N)) : 1.f;
            hE = hE + sv.W[(size_t)k * sv.wStride] * c;
        }
        return mask;
    }
    mask = 0u;
    many = true;
    // chunks of 8: the id and count loads of a chunk are in flight together
    for (int k0 = 0; k0 < (int)A.p.K; k0 += 8) {
        int id[8];
        unsigned c[8];
#pragma unroll
        for (int j = 0; j < 8; j++) id[j] = k0 + j < (int)A.p.K ? __ldg(sv.ids + (size_t)(k0 + j) * A.N) : 0;
#pragma unroll
        for (int j = 0; j < 8; j++) c[j] = k0 + j < (int)A.p.K ? __ldg(x + id[j]) : 0u;
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (c[j]) {
                hE = hE + sv.W[(size_t)(k0 + j) * sv.wStride] * (float)c[j];
                mask |= 1u << (k0 + j);
            }
    }
    return mask;
}

// The CTA's columns of the block's I -> all weights without their zeros, in shared memory: they are read
// between a step's spikes and the next step's threshold, where a read from L2 was a third of the
// step.  Per I neuron and 32 columns (a warp): the bits of the non-zero columns and the place of the first
// one's weight.  (hI is never -0, so leaving out the zeros does not change it.)
struct GabaView {
    const float *C;            // [nI][blockSize]
    const unsigned *bits;      // [nI][columns / 32], null: the weights did not fit, read C
    const unsigned *first;     // [nI][columns / 32]
    const float *w;
    int words;                 // columns / 32
};

// Builds it at dyn + A.gabaAt within A.gabaRoom bytes (every thread of the CTA calls it).
__device__ __forceinline__ GabaView stage_gaba(const AdjArgs &A, uint8_t *dyn, const float *C, int col0, AdjShared &sm) {
    GabaView v{C, nullptr, nullptr, nullptr, (int)blockDim.x / 32};
    const int words = v.words, cells = A.nI * words, bs = (int)A.p.blockSize;
    if (A.gabaAt < 0) return v;
    unsigned *bits = reinterpret_cast<unsigned *>(dyn + A.gabaAt), *first = bits + cells;
    float *w = reinterpret_cast<float *>(first + cells);
    const int cap = (A.gabaRoom - cells * 8) / 4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float *col = C + col0 + threadIdx.x;   // warp w holds column word w
    if (threadIdx.x == 0) sm.scan[0] = 0;
    __syncthreads();
    for (int p0 = 0; p0 < A.nI; p0 += 4) {
        float x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = p0 + u < A.nI ? __ldg(col + (size_t)(p0 + u) * bs) : 0.f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (p0 + u >= A.nI) break;
            const unsigned m = __ballot_sync(0xffffffffu, x[u] != 0.f);
            int at = 0;
            if (lane == 0) at = atomicAdd(&sm.scan[0], __popc(m));
            at = __shfl_sync(0xffffffffu, at, 0);
            const int k = (p0 + u) * words + warp;
            if (lane == 0) {
                bits[k] = m;
                first[k] = (unsigned)at;
            }
            const int mine = at + __popc(m & ((1u << lane) - 1u));
            if (x[u] != 0.f && mine < cap) w[mine] = x[u];
        }
    }
    __syncthreads();
    const bool fits = sm.scan[0] <= cap;
    __syncthreads();
    if (fits) {
        v.bits = bits;
        v.first = first;
        v.w = w;
    }
    return v;
}

// The weights of the block's spiking I neurons (ball: the step's ballots) onto this neuron, ascending.  Read
// from shared memory they are added to hI here; read from global memory, all but the last (up to)
// four are, and those are left in pend, to be added at the start of the next step, behind the
// work that does not need them.
struct Pending {
    float w[4];
    int n;
};

__device__ __forceinline__ void gaba_inputs(const AdjArgs &A, const GabaView &v, int local, const unsigned *ball, float &hI,
                                            Pending &pd) {
    const pv1_adj_problem &P = A.p;
    const int nWarp = ((int)P.blockSize + 31) / 32;
    const int lane = threadIdx.x & 31, w0 = (int)P.nE / 32;
    const unsigned mine = lane >= w0 && lane < nWarp ? ball[lane] : 0u;
    unsigned nz = __ballot_sync(0xffffffffu, mine != 0);
    pd.n = 0;
    if (!nz) return;
    unsigned cur = 0u;
    int w = 0;
    auto next = [&]() {   // the next spiking I neuron; only while there is one
        if (!cur) {
            w = __ffs(nz) - 1;
            nz &= nz - 1;
            cur = __shfl_sync(0xffffffffu, mine, w);
        }
        const int pre = w * 32 + __ffs(cur) - 1 - (int)P.nE;
        cur &= cur - 1;
        return pre;
    };
    if (v.bits) {
        const int word = threadIdx.x >> 5;
        while (nz | cur) {
            const int k = next() * v.words + word;
            const unsigned m = v.bits[k];
            if ((m >> lane) & 1u) hI = hI + v.w[v.first[k] + __popc(m & ((1u << lane) - 1u))];
        }
        return;
    }
    while (nz | cur) {
        // a full batch left from before is followed by more: add it
        if (pd.n == 4) {
#pragma unroll
            for (int j = 0; j < 4; j++) hI = hI + pd.w[j];
        }
        pd.n = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (!(nz | cur)) break;
            pd.w[j] = __ldg(v.C + (size_t)next() * P.blockSize + local);
            pd.n = j + 1;
        }
    }
}

__device__ __forceinline__ void add_pending(float &hI, Pending &pd) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (j >= pd.n) break;
        hI = hI + pd.w[j];
    }
    pd.n = 0;
}

// Copies the neuron's synapse weights into the CTA's shared memory (column per thread) where there is
// room for them.
__device__ __forceinline__ SynView stage_synapses(const AdjArgs &A, uint8_t *dyn, int n) {
    SynView sv{A.b.ids + n, A.b.W + n, A.N};
    if (A.wAt >= 0) {
        float *sW = reinterpret_cast<float *>(dyn + A.wAt);
        for (int k = 0; k < (int)A.p.K; k++) sW[k * blockDim.x + threadIdx.x] = __ldg(A.b.W + (size_t)k * A.N + n);
        sv.W = sW + threadIdx.x;
        sv.wStride = (int)blockDim.x;
    }
    return sv;
}

// Sets up the exchange of a CTA; every thread of the block's CTAs calls it once.
__device__ __forceinline__ void init_exchange(const AdjArgs &A, uint8_t *dyn, AdjShared &sm, int firstN) {
    unsigned *m = reinterpret_cast<unsigned *>(dyn + A.maskAt);
    if (threadIdx.x == 0) {
        for (int k = 0; k < 2; k++) {
            sm.mask[k] = m + k * blockDim.x;
            sm.many[k] = m + (2 + k) * blockDim.x;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&sm.bar[k])), "r"((int)A.p.blockSize / 32));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int k = 0; k < 4; k++) m[k * blockDim.x + threadIdx.x] = 0u;
    if (threadIdx.x < 64) sm.ball[threadIdx.x >> 5][threadIdx.x & 31] = 0u;
    __syncthreads();
    build_events(A, dyn, firstN, blockDim.x, sm);
    block_sync(A.split);   // every CTA of the block is set up before the first remote store
}

// The end of a CTA's exchanges: no CTA leaves while a peer's stores are on their way to it.
__device__ __forceinline__ void leave_exchange(AdjShared &sm, int split, unsigned phase, int lost) {
    if (split == 1) return;
    cg::this_cluster().sync();
    if (lost >= 0) wait_block(sm, lost, phase);   // what was late: everyone has sent by now
}

// One forward step of a neuron with its exchange: shared by the forward and the recompute of the
// backward.  vnext, spk, refr: the step's results; mask, many: its LGN events.
// lost: the parity of the exchange whose wait ran out, else -1.  From then on the warp neither sends nor
// waits, so that what is left takes no time and the peers' waits run out as well, once each; its
// potentials are NaN, which the outputs show.
struct StepOut {
    float vnext;
    bool spk, refr, many;
    unsigned mask;
};

__device__ __forceinline__ StepOut exchange_step(const AdjArgs &A, AdjShared &sm, AState &s, float I0, bool isE, int local,
                                                 const GabaView &gv, const uint8_t *x, int par, unsigned &phase,
                                                 const SynView &sv, Pending &pd, int &lost) {
    StepOut o;
    float gE1, hE1, gI1, hI1;
    o.vnext = adj_neuron_step(A.p, s, I0, isE, o.spk, o.refr, gE1, hE1, gI1, hI1);
    const unsigned bal = __ballot_sync(0xffffffffu, o.spk);
    if (lost < 0) {
        send_ballot(sm, par, local >> 5, bal, A.split);
        if (!wait_block(sm, par, phase)) lost = par;
    }
    if (lost >= 0) o.vnext = nanf("");
    o.mask = lgn_inputs(A, x, sm, par, hE1, sv, o.many);
    gaba_inputs(A, gv, local, sm.ball[par], hI1, pd);
    s.v = o.vnext;
    s.gE = gE1; s.hE = hE1; s.gI = gI1; s.hI = hI1;
    return o;
}

template <int MaxThreads>
__global__ void __launch_bounds__(MaxThreads, 1) adj_forward_kernel(AdjArgs A) {
    __shared__ AdjShared sm;
    extern __shared__ __align__(16) uint8_t dyn[];
    const pv1_adj_problem &P = A.p;
    const int split = A.split;
    const int blk = blockIdx.x / split, b = blockIdx.y;
    const int local = (blockIdx.x % split) * blockDim.x + threadIdx.x;
    const int n = blk * (int)P.blockSize + local;
    const size_t bn = (size_t)b * A.N + n;
    const bool isE = local < (int)P.nE;
    const float I0 = A.b.I0[n];
    const float *C = A.b.Crec + (size_t)blk * A.nI * P.blockSize;
    AState s{A.b.v0[bn], 0.f, 0.f, 0.f, 0.f, 0};
    float cnt = 0.f, vsum = 0.f;
    const size_t BN = (size_t)P.B * A.N;
    const uint8_t *row = A.b.X + (size_t)b * P.T * P.nLGN;
    init_exchange(A, dyn, sm, n - threadIdx.x);
    const SynView sv = stage_synapses(A, dyn, n);
    const GabaView gv = stage_gaba(A, dyn, C, local - threadIdx.x, sm);
    const bool fits = row_fits(A);
    RowShare share = fetch_row(A, row, fits);
    unsigned phase = 0u;
    int lost = -1;
    Pending pd;
    pd.n = 0;
    int toCk = 0, toWin = (int)P.win;
    float *ck = A.b.ck + bn;
    size_t o = (size_t)b * A.nWin * A.N + n;
    for (int t = 0; t < (int)P.T; t++, row += P.nLGN) {
        const int par = t & 1;
        mark_events(A, dyn, row, share, fits, sm, par);
        if (t + 1 < (int)P.T) share = fetch_row(A, row + P.nLGN, fits);
        add_pending(s.hI, pd);
        if (toCk == 0) {
            ck[0] = s.v; ck[BN] = s.gE; ck[2 * BN] = s.hE; ck[3 * BN] = s.gI; ck[4 * BN] = s.hI;
            ck[5 * BN] = (float)s.ref;
            ck += 6 * BN;
            toCk = (int)P.seg;
        }
        toCk--;
        const StepOut r = exchange_step(A, sm, s, I0, isE, local, gv, row, par, phase, sv, pd, lost);
        cnt += r.spk ? 1.f : 0.f;
        vsum += r.vnext;
        if (--toWin == 0) {
            A.b.rates[o] = cnt / ((float)P.win * P.dt * 1e-3f);
            A.b.vbar[o] = vsum / (float)P.win;
            o += A.N;
            cnt = 0.f;
            vsum = 0.f;
            toWin = (int)P.win;
        }
    }
    leave_exchange(sm, split, phase, lost);
}

__device__ __forceinline__ void block_add_double(double v, double *out, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < (blockDim.x + 31) / 32 ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) atomicAdd(out, v);
    }
}

constexpr int kScrWords = 7;   // v, gE, hE, gI, hI, flags, LGN event mask per neuron and step

// A neuron's recorded step: the state before it, flags (1: refractory, 2: spike, 4: some LGN count above
// 1) and LGN event mask.
struct Recorded {
    float v, gE, hE, gI, hI, flags;
    unsigned mask;
};

__device__ __forceinline__ Recorded load_recorded(const float *o, int bs) {
    return Recorded{o[0], o[bs], o[2 * bs], o[3 * bs], o[4 * bs], o[5 * bs], __float_as_uint(o[6 * bs])};
}

template <int MaxThreads>
__global__ void __launch_bounds__(MaxThreads, 1) adj_backward_kernel(AdjArgs A) {
    __shared__ AdjShared sm;
    __shared__ float lam[1024];
    __shared__ float dS[1024];
    __shared__ double red[32];
    extern __shared__ __align__(16) uint8_t dyn[];
    const pv1_adj_problem &P = A.p;
    const int split = A.split;
    const int ctaN = (int)blockDim.x;
    const int blk = blockIdx.x / split, b = blockIdx.y;
    const int local = (blockIdx.x % split) * ctaN + threadIdx.x;
    const int bs = (int)P.blockSize;
    const int n = blk * bs + local;
    const size_t bn = (size_t)b * A.N + n;
    const bool isE = local < (int)P.nE;
    const float I0 = A.b.I0[n];
    const size_t BN = (size_t)P.B * A.N;
    float *scr = A.b.scratch + (size_t)(b * (int)P.nblock + blk) * P.seg * kScrWords * bs + local;
    const size_t scrStep = (size_t)kScrWords * bs;
    const float *C = A.b.Crec + (size_t)blk * A.nI * bs;
    const float rateScale = 1.f / ((float)P.win * P.dt * 1e-3f);
    const float invWin = 1.f / (float)P.win;
    const int warp = local >> 5, lane = local & 31, nWarp = (bs + 31) / 32;
    const uint8_t *Xb = A.b.X + (size_t)b * P.T * P.nLGN;
    init_exchange(A, dyn, sm, n - threadIdx.x);
    const SynView sv = stage_synapses(A, dyn, n);
    const GabaView gv = stage_gaba(A, dyn, C, local - threadIdx.x, sm);
    const bool fits = row_fits(A);
    unsigned phase = 0u;
    int par = 0;   // of the next exchange
    int lost = -1;
    Pending pd;
    pd.n = 0;
    // adjoints of the state after the current step
    float lv = 0.f, lgE = 0.f, lhE = 0.f, lgI = 0.f, lhI = 0.f;
    float dEdE = 0.f, dErE = 0.f, ddodE = 0.f, dEdI = 0.f, dErI = 0.f, ddodI = 0.f;
    // the current window's share of the loss gradient
    int inWin = 0;
    size_t oo = ((size_t)b * A.nWin + A.nWin) * A.N + n;
    float gR = 0.f, gV = 0.f;
    for (int sg = A.nSeg - 1; sg >= 0; sg--) {
        const int t0 = sg * (int)P.seg;
        const int t1 = min((int)P.T, t0 + (int)P.seg);
        // recompute the segment forward from its checkpoint
        const float *ck = A.b.ck + (size_t)sg * 6 * BN + bn;
        AState s{ck[0], ck[BN], ck[2 * BN], ck[3 * BN], ck[4 * BN], (int)ck[5 * BN]};
        const uint8_t *row = Xb + (size_t)t0 * P.nLGN;
        RowShare share = fetch_row(A, row, fits);
        float *o = scr;
        for (int t = t0; t < t1; t++, row += P.nLGN, o += scrStep, par ^= 1) {
            mark_events(A, dyn, row, share, fits, sm, par);
            if (t + 1 < t1) share = fetch_row(A, row + P.nLGN, fits);
            add_pending(s.hI, pd);
            o[0] = s.v; o[bs] = s.gE; o[2 * bs] = s.hE; o[3 * bs] = s.gI; o[4 * bs] = s.hI;
            const StepOut r = exchange_step(A, sm, s, I0, isE, local, gv, row, par, phase, sv, pd, lost);
            o[5 * bs] = (float)((r.refr ? 1 : 0) | (r.spk ? 2 : 0) | (r.many ? 4 : 0));
            o[6 * bs] = __uint_as_float(r.mask);
        }
        pd.n = 0;
        // adjoint backwards through the segment; a step's record is fetched while the one after it is
        // worked on (without that its seven loads were half of the step)
        o -= scrStep;
        Recorded next = load_recorded(o, bs);
        for (int t = t1 - 1; t >= t0; t--) {
            const Recorded q = next;
            if (t > t0) {
                o -= scrStep;
                next = load_recorded(o, bs);
            }
            // recurrent term: dS[p] = sum_n C[p][n] * lambda_hI(t+1)[n] for the I neurons p
            if (P.recGrad) {
                share_float(&lam[local], lhI, split);
                block_sync(split);
                for (int p0 = warp * 4; p0 < A.nI; p0 += nWarp * 4) {
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    const float *r0 = C + (size_t)p0 * bs;
                    for (int j = lane; j < bs; j += 32) {
                        const float l = lam[j];
#pragma unroll
                        for (int u = 0; u < 4; u++) acc[u] += __ldg(r0 + (size_t)u * bs + j) * l;
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        for (int x = 16; x > 0; x >>= 1) acc[u] += __shfl_down_sync(0xffffffffu, acc[u], x);
                        // into the CTA that holds I neuron p
                        if (lane == 0) store_at_rank(&dS[p0 + u], acc[u], ((int)P.nE + p0 + u) / ctaN, split);
                    }
                }
                block_sync(split);   // dS is there; everyone has read lam
            }
            if (inWin == 0) {
                inWin = (int)P.win;
                oo -= A.N;
                gR = A.b.gR ? A.b.gR[oo] * rateScale : 0.f;
                gV = A.b.gV ? A.b.gV[oo] * invWin : 0.f;
            }
            inWin--;
            const float v = q.v, gE = q.gE, hE = q.hE, gI = q.gI, hI = q.hI;
            const int fl = (int)q.flags;
            float dLds = gR;
            if (!isE && P.recGrad) dLds += dS[local - (int)P.nE];
            float lvn_next = lv + gV;   // adjoint of v(t+1)
            // LGN weight gradients at this step's events (the recompute recorded which synapses)
            for (unsigned mask = q.mask; mask; mask &= mask - 1) {
                const int k = __ffs(mask) - 1;
                const float c =
                    fl & 4 ? (float)__ldg(Xb + (size_t)t * P.nLGN + __ldg(sv.ids + (size_t)k * A.N)) : 1.f;
                atomicAdd(A.b.gW + (size_t)k * A.N + n, lhE * c);
            }
            const bool refr = fl & 1, spk = fl & 2;
            const float gE1 = gE * P.EdE + hE * P.dodE * (P.EdE - P.ErE);
            const float gI1 = gI * P.EdI + hI * P.dodI * (P.EdI - P.ErI);
            float lgE1 = lgE, lgI1 = lgI;
            const float lhE1 = lhE, lhI1 = lhI;
            float lvt = 0.f, lgE0 = 0.f, lgI0 = 0.f;
            if (!refr) {
                const float k1 = adj_f(v, gE, gI, P.gL, P.vL, P.vE, P.vI, I0);
                const float v1 = v + P.dt * k1;
                const float k2 = adj_f(v1, gE1, gI1, P.gL, P.vL, P.vE, P.vI, I0);
                const float vn = v + (P.dt * 0.5f) * (k1 + k2);
                const float xsv = vn - P.vThres;
                const float den = 1.f + P.slope * fabsf(xsv);
                const float lvn = (spk ? 0.f : lvn_next) + pv1::div_sparse(dLds, den * den);
                const float lk2 = lvn * (P.dt * 0.5f);
                const float a1 = -P.gL - gE1 - gI1;
                const float lv1 = lk2 * a1;
                const float lk1 = lvn * (P.dt * 0.5f) + lv1 * P.dt;
                const float a0 = -P.gL - gE - gI;
                lvt = lvn + lk1 * a0 + lv1;
                lgE0 = -lk1 * (v - P.vE);
                lgI0 = -lk1 * (v - P.vI);
                lgE1 += -lk2 * (v1 - P.vE);
                lgI1 += -lk2 * (v1 - P.vI);
            }
            dEdE += lgE1 * (gE + hE * P.dodE);
            ddodE += lgE1 * hE * (P.EdE - P.ErE);
            dErE += lhE1 * hE - lgE1 * hE * P.dodE;
            dEdI += lgI1 * (gI + hI * P.dodI);
            ddodI += lgI1 * hI * (P.EdI - P.ErI);
            dErI += lhI1 * hI - lgI1 * hI * P.dodI;
            lgE = lgE1 * P.EdE + lgE0;
            lhE = lgE1 * P.dodE * (P.EdE - P.ErE) + lhE1 * P.ErE;
            lgI = lgI1 * P.EdI + lgI0;
            lhI = lgI1 * P.dodI * (P.EdI - P.ErI) + lhI1 * P.ErI;
            lv = lvt;
        }
    }
    block_add_double(dEdE, A.b.gC + 0, red);
    block_add_double(dErE, A.b.gC + 1, red);
    block_add_double(ddodE, A.b.gC + 2, red);
    block_add_double(dEdI, A.b.gC + 3, red);
    block_add_double(dErI, A.b.gC + 4, red);
    block_add_double(ddodI, A.b.gC + 5, red);
    leave_exchange(sm, split, phase, lost);
}

int adj_check(const pv1_adj_problem *p, const pv1_adj_buffers *b, AdjArgs *A, bool backward) {
    if (!p || !b) return PV1_E_ARG;
    if (p->blockSize < 32 || p->blockSize > 1024 || p->blockSize % 32 || p->nE % 32 || p->nE >= p->blockSize ||
        p->B < 1 || p->nblock < 1 || p->K < 1 || p->K > kAdjMaxK || p->T < 1 || p->seg < 1 || p->win < 1 ||
        p->T % p->win || p->nLGN < 1 || !(p->dt > 0)) {
        g_adjErr = "bad problem sizes (blockSize multiple of 32 up to 1024, nE multiple of 32, K <= 32, "
                   "T a multiple of win)";
        return PV1_E_ARG;
    }
    if (!b->ids || !b->W || !b->X || !b->Crec || !b->I0 || !b->v0 || !b->ck) {
        g_adjErr = "missing input buffer";
        return PV1_E_ARG;
    }
    if (!backward && (!b->rates || !b->vbar)) {
        g_adjErr = "missing output buffer";
        return PV1_E_ARG;
    }
    if (backward && (!b->gW || !b->gC || !b->scratch)) {
        g_adjErr = "missing gradient or scratch buffer";
        return PV1_E_ARG;
    }
    A->p = *p;
    A->b = *b;
    A->N = (int)(p->nblock * p->blockSize);
    A->nI = (int)(p->blockSize - p->nE);
    A->nWin = (int)(p->T / p->win);
    A->nSeg = (int)((p->T + p->seg - 1) / p->seg);
    // CTAs per block where the caller leaves it open.  Two halve a step's work per SM and cost an exchange
    // over the cluster: measured forward and backward of 480 steps without the recurrent term, one CTA
    // against two: 128 neurons 1,981 and 2,057 us, 256 neurons 2,245 and 2,163, 1,024 neurons 4,449 and
    // 3,125.  With it the backward exchanges every step's adjoints: 128 neurons 2,455 and 4,431, 1,024
    // neurons 9,687 and 15,865.
    int split = (int)p->ctaSplit;
    if (split == 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const bool wide = p->blockSize >= 256 && p->blockSize % 64 == 0 && !(backward && p->recGrad);
        split = (wide && (long long)p->B * p->nblock * 2 <= sms) ? 2 : 1;
    }
    if (split != 1 && (split != 2 || p->blockSize % 64)) {
        g_adjErr = "ctaSplit must be 0, 1 or 2 (2 needs blockSize a multiple of 64)";
        return PV1_E_ARG;
    }
    A->split = split;
    return PV1_OK;
}

// Dynamic shared memory: the masks, the event lists if they fit, then the weights if they fit.
constexpr size_t kAdjRoom = 200 * 1024;
void adj_smem_plan(AdjArgs &A) {
    const int threads = (int)(A.p.blockSize / A.split);
    const size_t room = kAdjRoom;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        if (at + bytes > room) return -1;
        const int where = (int)at;
        at = (at + bytes + 15) / 16 * 16;
        return where;
    };
    A.maskAt = take((size_t)4 * threads * sizeof(unsigned));
    const size_t off = ((size_t)A.p.nLGN + 1) * sizeof(unsigned), ent = (size_t)A.p.K * threads * sizeof(unsigned short);
    A.offAt = A.entAt = -1;
    if (at + off + 16 + ent <= room) {
        A.offAt = take(off);
        A.entAt = take(ent);
    }
    A.wAt = take((size_t)A.p.K * threads * sizeof(float));
    // the rest, as far as the weights could need it, for the inhibitory ones
    const size_t words = (size_t)A.nI * (threads / 32) * 8, all = words + (size_t)A.nI * threads * sizeof(float);
    const size_t rest = std::min(room - at, all);
    A.gabaAt = -1;
    A.gabaRoom = 0;
    if (rest > words + all / 16) {
        A.gabaRoom = (int)rest;
        A.gabaAt = take(rest);
    }
    A.smemBytes = (int)at;
}

template <class Kern>
cudaError_t adj_launch(Kern kern, const AdjArgs &A, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(A.p.nblock * A.split, A.p.B);
    cfg.blockDim = dim3(A.p.blockSize / A.split);
    cfg.dynamicSmemBytes = (size_t)A.smemBytes;
    // the same limit for every problem: it belongs to the kernel, and another thread may be about to launch it
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAdjRoom);
    if (e != cudaSuccess) return e;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = A.split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = A.split > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, A);
}

}  // namespace

extern "C" {

const char *pv1_adj_last_error(void) { return g_adjErr.c_str(); }

uint64_t pv1_adj_checkpoint_floats(const pv1_adj_problem *p) {
    if (!p) return 0;
    return (uint64_t)((p->T + p->seg - 1) / p->seg) * 6 * p->B * p->nblock * p->blockSize;
}

uint64_t pv1_adj_scratch_floats(const pv1_adj_problem *p) {
    if (!p) return 0;
    return (uint64_t)p->B * p->nblock * p->seg * kScrWords * p->blockSize;
}

int pv1_adj_forward(const pv1_adj_problem *p, const pv1_adj_buffers *b, void *stream) {
    AdjArgs A;
    int r = adj_check(p, b, &A, false);
    if (r) return r;
    adj_smem_plan(A);
    cudaError_t e = A.p.blockSize / A.split <= 512 ? adj_launch(adj_forward_kernel<512>, A, (cudaStream_t)stream)
                                                   : adj_launch(adj_forward_kernel<1024>, A, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        g_adjErr = cudaGetErrorString(e);
        return PV1_E_CUDA;
    }
    return PV1_OK;
}

int pv1_adj_backward(const pv1_adj_problem *p, const pv1_adj_buffers *b, void *stream) {
    AdjArgs A;
    int r = adj_check(p, b, &A, true);
    if (r) return r;
    adj_smem_plan(A);
    cudaError_t e = A.p.blockSize / A.split <= 512 ? adj_launch(adj_backward_kernel<512>, A, (cudaStream_t)stream)
                                                   : adj_launch(adj_backward_kernel<1024>, A, (cudaStream_t)stream);
    if (e != cudaSuccess) {
        g_adjErr = cudaGetErrorString(e);
        return PV1_E_CUDA;
    }
    return PV1_OK;
}

}  // extern "C"
