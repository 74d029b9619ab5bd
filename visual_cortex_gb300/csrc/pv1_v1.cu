// V1 stage of the patchV1 hot path on GB300 (sm_103a).
//
// The reference runs, per step, compute_V_collect_spike_learnFF_fast (src/coredynamics.cu:
// 1235-2059), then recal_G_mat_nd_fast for the near-neighbour blocks (:2609-2922), then a
// single-threaded host loop for the far synapses (recal_G_vec :181-372, fill_fSpikeTrain
// src/stats.cu:114-126) whose result is copied back and added by sum_G (:2312-2349).
//
// Here every simulation step has three phases, one thread per neuron:
//   A. deliver the previous step's spikes: every CTA compacts the spikers of its neighbour
//      blocks with warp ballots (ascending neuron order, E before I), stages their unit
//      conductance (og/oh) in shared memory and reads one coalesced conMat row per spiker;
//      far events that arrive in the previous step come from a fixed-point ring filled by
//      phase C.  The sum is added to g/h exactly where the reference's delivery adds it.
//   B. the V1 membrane step (conductance decay, LGN input, RK2 AdEx/LIF, spike-time
//      interpolation, refractoriness), with the float operations of the reference's kernel.
//   C. push this step's spikes into the far-delivery ring: one event per (spike, far
//      synapse), with the reference's delay arithmetic deciding the arrival step.
// Adding the previous step's delivery before this step's decay is the same sequence of
// float operations as the reference's separate kernels.
//
// v1_step_kernel runs these phases one step per launch (state in HBM).  v1_persistent_kernel and, for the
// trials of a sweep, v1_batch_persistent_kernel run K steps in one launch with the neuron state and the
// generators in registers and the LGN synapses in shared memory.  All are instantiated with and without the random-number paths (noise, synaptic
// failure); the host picks the variant.  Per-species arrays use compile-time indices so that
// they stay in registers.
#include <algorithm>
#include "pv1_internal.cuh"
#include "pv1_rng.cuh"

namespace pv1 {

constexpr int kCta = 256;
constexpr int kWarps = kCta / 32;
constexpr int kMaxBS = 1024;
constexpr int kLgnBatch = 8;
constexpr int kMaxLgnReg = 32;        // LGN synapses kept in shared memory by the persistent kernel
// The same in the batched persistent kernel, and the words of an LGN row's spike bits: with PShared
// and the trial block its shared memory still fits an SM twice.
constexpr int kBatchLgn = 24;
constexpr int kBatchBits = 512;
constexpr size_t kBatchDyn = ((size_t)2 * kBatchLgn * kCta + 2 * kBatchBits) * sizeof(float);
constexpr int kConBatch = 8;          // conMat rows fetched together

__device__ __forceinline__ int type_of(const V1Params &P, int local) {
    int t = P.nType - 1;
#pragma unroll
    for (int j = kMaxType - 1; j >= 0; j--) {
        if (j < P.nType && local < P.typeAcc[j]) t = j;
    }
    return t;
}

// Record offsets inside one rawData record (src/patch.cu:6138-6165, src/stats.cu:39-97).
struct RecOff {
    long long sinfo, dep, w, v, gFF, hFF, gE, gI, hE, hI;
};
__device__ __forceinline__ RecOff rec_off(const V1Params &P) {
    RecOff o;
    long long n = P.nV1;
    o.sinfo = 0;
    o.dep = n;
    o.w = 2 * n;
    o.v = (2 + (P.iModel == 1)) * n;
    o.gFF = o.v + n;
    o.hFF = o.gFF + P.ngFF * n;
    o.gE = o.hFF + (P.hWrite ? P.ngFF * n : 0);
    o.gI = o.gE + P.ngE * n;
    o.hE = o.gI + P.ngI * n;
    o.hI = o.hE + P.ngE * n;
    return o;
}

// Per-neuron dynamic state (registers).
struct NState {
    float v, w, tBack, lastNoise;
    float gE[kMaxNG], hE[kMaxNG], gI[kMaxNG], hI[kMaxNG], gFF[kMaxNG], hFF[kMaxNG];
};

// Barrier among the CTA's kCta neuron threads (a persistent CTA can hold push warps beside them).
__device__ __forceinline__ void neuron_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCta) : "memory"); }

// Staging of the general near delivery: the spikers of one neighbour block.
struct Smem {
    int pre[kMaxBS];
    float og[kMaxNG][kMaxBS];
    float oh[kMaxNG][kMaxBS];
    unsigned ball[kMaxBS / 32];
};

__device__ __forceinline__ void load_state(const V1Params &P, int i, NState &s) {
    const int nV1 = P.nV1;
    s.v = P.v[i];
    s.w = P.iModel == 1 ? P.w[i] : 0.0f;
    s.tBack = P.tBack[i];
    s.lastNoise = P.tau_noise > 0 ? P.lastNoise[i] : 0.f;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        s.gE[ig] = ig < P.ngE ? P.gE[ig * nV1 + i] : 0.f;
        s.hE[ig] = ig < P.ngE ? P.hE[ig * nV1 + i] : 0.f;
        s.gI[ig] = ig < P.ngI ? P.gI[ig * nV1 + i] : 0.f;
        s.hI[ig] = ig < P.ngI ? P.hI[ig * nV1 + i] : 0.f;
        s.gFF[ig] = ig < P.ngFF ? P.gFF[ig * nV1 + i] : 0.f;
        s.hFF[ig] = ig < P.ngFF ? P.hFF[ig * nV1 + i] : 0.f;
    }
}

__device__ __forceinline__ void store_state(const V1Params &P, int i, const NState &s) {
    const int nV1 = P.nV1;
    P.v[i] = s.v;
    if (P.iModel == 1) P.w[i] = s.w;
    P.tBack[i] = s.tBack;
    if (P.tau_noise > 0) P.lastNoise[i] = s.lastNoise;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < P.ngE) { P.gE[ig * nV1 + i] = s.gE[ig]; P.hE[ig * nV1 + i] = s.hE[ig]; }
        if (ig < P.ngI) { P.gI[ig * nV1 + i] = s.gI[ig]; P.hI[ig * nV1 + i] = s.hI[ig]; }
        if (ig < P.ngFF) { P.gFF[ig * nV1 + i] = s.gFF[ig]; P.hFF[ig * nV1 + i] = s.hFF[ig]; }
    }
}

// Compacts the spike words blk[0..bs) that are >= 1 into sm.pre[] (ascending index) and
// stages the unit conductance of each (output_g/h of compute_V, src/coredynamics.cu:
// 2008-2041) in sm.og/sm.oh.  Returns the count; *cntE receives the number of excitatory
// spikers (index < nE), which come first.  Three CTA barriers when there are spikers, two
// otherwise.
__device__ __forceinline__ int compact_spikers(const V1Params &P, const float *__restrict__ blk, Smem &sm,
                                               int *cntE) {
    const int bs = P.blockSize, nE = P.nE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (bs + 31) >> 5;
    const float dt = P.dt;
    float vals[kMaxBS / kCta];
#pragma unroll
    for (int k = 0; k < kMaxBS / kCta; k++) {
        const int j = k * kCta + threadIdx.x;
        vals[k] = j < bs ? __ldcg(blk + j) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kMaxBS / kCta; k++) {
        const int j = k * kCta + threadIdx.x;
        const bool f = j < bs && vals[k] >= 1.0f;
        const unsigned bal = __ballot_sync(0xffffffffu, f);
        if (k * kCta < bs && lane == 0) sm.ball[k * kWarps + warp] = bal;
    }
    neuron_sync();
    // every warp scans the block's ballot words itself (no second barrier): lane l holds word l
    const unsigned wb = lane < nw ? sm.ball[lane] : 0u;
    const int c = __popc(wb);
    int below = 0;
    if ((lane + 1) * 32 <= nE) below = c;
    else if (lane * 32 < nE) below = __popc(wb & ((1u << (nE - lane * 32)) - 1u));
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    *cntE = below;
    if (total == 0) return 0;
    const int excl = incl - c;
#pragma unroll
    for (int k = 0; k < kMaxBS / kCta; k++) {
        const int j = k * kCta + threadIdx.x;
        // word k * kWarps + warp holds this warp's lanes for pass k (j >> 5)
        const int wbase = __shfl_sync(0xffffffffu, excl, (k * kWarps + warp) & 31);
        const unsigned wbits = __shfl_sync(0xffffffffu, wb, (k * kWarps + warp) & 31);
        if (j < bs && vals[k] >= 1.0f) {
            const int pos = wbase + __popc(wbits & ((1u << lane) - 1u));
            sm.pre[pos] = j;
            const float sI = vals[k];
            const float nsp = floorf(sI);
            const float tsp = (sI - nsp) * dt;
            const bool isE = j < nE;
#pragma unroll
            for (int ig = 0; ig < kMaxNG; ig++) {
                if (ig < (isE ? P.ngE : P.ngI)) {
                    float g = 0.f, h = 0.f;
                    if (isE) cond_input(P.condE, g, h, nsp, dt - tsp, ig);
                    else cond_input(P.condI, g, h, nsp, dt - tsp, ig);
                    sm.og[ig][pos] = g;
                    sm.oh[ig][pos] = h;
                }
            }
        }
    }
    neuron_sync();
    return total;
}

__device__ __forceinline__ void prefetch_far(const V1Params &P, int e0, int deg) {
    const unsigned bytes = (unsigned)deg * 16u;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(P.farRec + e0), "r"(bytes) : "memory");
}

// Sends to L2 what is read when neuron i (local index `local` of block b) spikes: its rows of the near
// tiles that list block b (read by the delivery, whole 16-byte aligned rows), and the whole
// 16-byte chunks of `farDeg` synapses of its far list (read by the push).  Hints only: nothing
// waits on them.
__device__ __forceinline__ void prefetch_spiker(const V1Params &P, int b, int local, int farE0, int farDeg) {
    if (P.noDelay && P.nearRevOff && (P.blockSize & 3) == 0) {
        const unsigned bytes = (unsigned)P.blockSize * 4u;
        for (int e = __ldg(P.nearRevOff + b); e < __ldg(P.nearRevOff + b + 1); e++) {
            const float *row = P.conMat + ((size_t)__ldg(P.nearRev + e) * P.blockSize + local) * P.blockSize;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row), "r"(bytes) : "memory");
        }
    }
    if (farDeg > 0) prefetch_far(P, farE0, farDeg);
}

// The excitatory filtered rate of learning 1, 2 and 4, advanced over step tp in the near
// delivery as recal_G_mat_nd_fast does (src/coredynamics.cu:2866-2890): from the value stored
// at the spike time when the neuron spiked (slot 1), else the step start (slot 0), plus the
// spike count, decayed over the rest of the step with the cortical E types' tauAvg.
__device__ __forceinline__ void learn_avg_delivery(const V1Params &P, float postSInfo, const float *avg0, const float *avg1,
                                                   float *out) {
    const float dt = P.dt;
    const float postNsp = floorf(postSInfo);
    const float postTsp = postSInfo > 0 ? postSInfo - postNsp : 1.f;
    float lAvgE = postNsp > 0 ? *avg1 : *avg0;
    float delta_t = dt;
    if (postNsp > 0) delta_t = dt * (1 - postTsp);
    lAvgE += postNsp;
    lAvgE *= expf(-delta_t / P.tauAvgCortical);
    *out = lAvgE;
}

// Ring slot of step t in the far/near event rings.
__device__ __forceinline__ int far_ring_slot(const V1Params &P, long long t) {
    const long long r = t % P.farDepth;
    return (int)(r < 0 ? r + P.farDepth : r);
}

// Far events of one ring slot for one neuron, and whether a far presynaptic neuron spiked in
// that step (the reference delivers far input only then).
struct FarIn {
    unsigned long long g[2 * kMaxNG], h[2 * kMaxNG];
    bool spiked;
};

__device__ __forceinline__ void far_fetch(const V1Params &P, int farSlot, int flagSlot, int i, FarIn &f) {
    const int ns = P.ngE + P.ngI, nV1 = P.nV1;
    const unsigned long long *acc = P.farAcc + (size_t)farSlot * ns * 2 * nV1;
    f.spiked = __ldcg(P.farFlag + flagSlot) != 0;
#pragma unroll
    for (int q = 0; q < 2 * kMaxNG; q++) {
        f.g[q] = q < ns ? __ldcg(acc + (size_t)(2 * q) * nV1 + i) : 0ull;
        f.h[q] = q < ns ? __ldcg(acc + (size_t)(2 * q + 1) * nV1 + i) : 0ull;
    }
}

// Adds fetched far events to the conductances and clears the ring entries they came from.
__device__ __forceinline__ void far_apply(const V1Params &P, int farSlot, int i, const FarIn &f, NState &st) {
    const int ns = P.ngE + P.ngI, nV1 = P.nV1;
    unsigned long long *acc = P.farAcc + (size_t)farSlot * ns * 2 * nV1;
#pragma unroll
    for (int q = 0; q < 2 * kMaxNG; q++) {
        if (q < ns) {
            if (f.g[q] | f.h[q]) {
                acc[(size_t)(2 * q) * nV1 + i] = 0ull;
                acc[(size_t)(2 * q + 1) * nV1 + i] = 0ull;
            }
            if (f.spiked) {
                const float fg = far_from_fixed(f.g[q]);
                const float fh = far_from_fixed(f.h[q]);
#pragma unroll
                for (int ig = 0; ig < kMaxNG; ig++) {
                    if (q < P.ngE && ig == q) { st.gE[ig] += fg; st.hE[ig] += fh; }
                    if (q >= P.ngE && ig == q - P.ngE) { st.gI[ig] += fg; st.hI[ig] += fh; }
                }
            }
        }
    }
}

// Delayed near events (noDelay = 0) of one ring slot: taken into lg/lh, entries cleared.
__device__ __forceinline__ void near_ring_take(const V1Params &P, int farSlot, int i, float *lgE, float *lhE,
                                               float *lgI, float *lhI) {
    const int ns = P.ngE + P.ngI, nV1 = P.nV1, ngE = P.ngE;
    unsigned long long *nacc = P.nearAcc + (size_t)farSlot * ns * 2 * nV1;
#pragma unroll
    for (int q = 0; q < 2 * kMaxNG; q++) {
        if (q < ns) {
            unsigned long long *pg = nacc + (size_t)(2 * q) * nV1 + i;
            unsigned long long *ph = nacc + (size_t)(2 * q + 1) * nV1 + i;
            const unsigned long long ug = __ldcg(pg), uh = __ldcg(ph);
            if (ug | uh) {
                *pg = 0ull;
                *ph = 0ull;
                const float fg = far_from_fixed(ug), fh = far_from_fixed(uh);
#pragma unroll
                for (int ig = 0; ig < kMaxNG; ig++) {
                    if (q < ngE && ig == q) { lgE[ig] = fg; lhE[ig] = fh; }
                    if (q >= ngE && ig == q - ngE) { lgI[ig] = fg; lhI[ig] = fh; }
                }
            }
        }
    }
}

// The conductances of a step's record (ring slot recSlot), complete once its spikes are delivered.
__device__ __forceinline__ void record_conductances(const V1Params &P, int recSlot, int i, const NState &st) {
    const int nV1 = P.nV1;
    float *r = P.rec + recSlot * P.recStride;
    const RecOff o = rec_off(P);
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < P.ngE) r[o.gE + ig * nV1 + i] = st.gE[ig];
        if (ig < P.ngI) r[o.gI + ig * nV1 + i] = st.gI[ig];
        if (P.hWrite) {
            if (ig < P.ngE) r[o.hE + ig * nV1 + i] = st.hE[ig];
            if (ig < P.ngI) r[o.hI + ig * nV1 + i] = st.hI[ig];
        }
    }
}

// Failure draw of one near synapse from the spiker of rank `rank` among its block's E or I
// spikers: the pre type comes from that rank, as the reference takes it
// (src/coredynamics.cu:2760-2766, 2815-2821).
__device__ __forceinline__ float near_failure(const V1Params &P, float strength, bool isE, int rank, int itype,
                                              curandStateMRG32k3a &condState, float *recNear, int &nDraw) {
    const int ja = isE ? 0 : P.nTypeE, jb = isE ? P.nTypeE : P.nType;
    int jtype = ja;
    for (int jj = ja; jj < jb; jj++) {
        if (rank < P.typeAcc[jj]) { jtype = jj; break; }
    }
    const int idx = jtype * P.nType + itype;
    const float lp = P.synFail[idx];
    const float normed_std = sqrtf(lp * (1 - lp) / P.synPerCon[idx]);
    const float rnd = curand_normal(&condState);
    if (recNear) {
        if (nDraw < P.recCap) recNear[nDraw] = rnd;
        else atomicOr(P.err, kErrRecordOverflow);
    }
    nDraw++;
    return strength * (1 - lp + normed_std * rnd);
}

// Phase A: delivery of step tp's spikes to this thread's neuron (all kCta neuron threads of the
// CTA must call it; `active` masks the neuron work): any list of neighbour blocks, the spike
// words read from global memory.
template <bool Rng>
__device__ __forceinline__ void deliver_prev(const V1Params &P, long long tp, int b, int local, int i,
                                             bool active, int itype, NState &st,
                                             curandStateMRG32k3a &condState, Smem &sm, int farSlot = -1) {
    const int bs = P.blockSize, nV1 = P.nV1;
    // the far ring slot of step tp (tp mod farDepth; passed in by the persistent kernel)
    if (farSlot < 0 && P.farOn) farSlot = far_ring_slot(P, tp);
    const int ngE = P.ngE, ngI = P.ngI;
    const float *sPrev = P.sInfo + (size_t)(tp & 1) * nV1;
    float lgE[kMaxNG], lhE[kMaxNG], lgI[kMaxNG], lhI[kMaxNG], ipE[kMaxNG], ipI[kMaxNG];
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        lgE[ig] = lhE[ig] = lgI[ig] = lhI[ig] = 0.f;
        ipE[ig] = ig < ngE ? P.pE[itype * ngE + ig] : 0.f;
        ipI[ig] = ig < ngI ? P.pI[itype * ngI + ig] : 0.f;
    }
    // far events arriving in step tp, fetched early so that the loads overlap the compaction
    const int ns = ngE + ngI;
    const bool far = P.farClass && active;
    FarIn fin;
    if (far) far_fetch(P, farSlot, (int)((tp + 3) % 3), i, fin);
    float *recNear = nullptr;
    int nNearDraw = 0;
    if (Rng && P.recNear && active) {
        long long rs = tp - P.recStep0;
        if (rs >= 0 && rs < P.recSteps) recNear = P.recNear + ((size_t)rs * nV1 + i) * P.recCap;
    }
    // delayed near events with synaptic failure: recal_G_mat (src/coredynamics.cu:2138-2224)
    // restated per post -- its near synapses in the reference's order, the two spike-word
    // slots that can deliver in step tp, a normal draw from the post's generator for each
    // arriving event of a pair with failure rate p > 0, float sums in that order
    if constexpr (Rng) {
        if (P.nearPullOn && active) {
            const float dt = P.dt;
            for (int e = P.npOff[i]; e < P.npOff[i + 1]; e++) {
                const int pre = P.npPre[e];
                const int steps = P.npSteps[e];
                const float frac = P.npFrac[e];
                const bool preE = (pre % bs) < P.nE;
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const long long ts = tp - steps + k;
                    const long long row = ((ts % P.sDepth) + P.sDepth) % P.sDepth;
                    const float sI = __ldcg(P.sRing + (size_t)row * nV1 + pre);
                    if (!(sI >= 1.0f)) continue;
                    const float nsp = floorf(sI);
                    const float dtsp = (sI - nsp + (float)k) * dt - frac;
                    if (!(dtsp < dt && dtsp >= 0)) continue;
                    float f = P.npStr[e];
                    const float pf = P.npP[e];
                    if (pf > 0) {
                        const float rnd = curand_normal(&condState);
                        if (recNear) {
                            if (nNearDraw < P.recCap) recNear[nNearDraw] = rnd;
                            else atomicOr(P.err, kErrRecordOverflow);
                        }
                        nNearDraw++;
                        f *= 1 - pf + P.npStd[e] * rnd;
                    }
                    if (f > 0) {
                        const float delta = dt - dtsp;
#pragma unroll
                        for (int ig = 0; ig < kMaxNG; ig++) {
                            if (preE && ig < ngE)
                                cond_input(P.condE, lgE[ig], lhE[ig], nsp * f * ipE[ig], delta, ig);
                            if (!preE && ig < ngI)
                                cond_input(P.condI, lgI[ig], lhI[ig], nsp * f * ipI[ig], delta, ig);
                        }
                    }
                }
            }
        }
    }
    // delayed near events (noDelay = 0): recal_G_mat sums them into the same step's
    // conductance update; here they were pushed into their own ring
    if (!P.noDelay && P.nearOn && active) near_ring_take(P, farSlot, i, lgE, lhE, lgI, lhI);
    const int nnb = P.noDelay ? P.nNearNB[b] : 0;
    for (int ib = 0; ib < nnb; ib++) {
        const int nb = P.nbId[b * P.nnbMax + ib];
        int cntE;
        const int cnt = compact_spikers(P, sPrev + (size_t)nb * bs, sm, &cntE);
        if (cnt == 0) continue;
        if (active) {
            const float *col = P.conMat + ((size_t)(b * P.nnbMax + ib) * bs) * bs + local;
            for (int r0 = 0; r0 < cnt; r0 += kConBatch) {
                float sv[kConBatch];
#pragma unroll
                for (int k = 0; k < kConBatch; k++)
                    sv[k] = r0 + k < cnt ? __ldg(col + (size_t)sm.pre[r0 + k] * bs) : 0.f;
#pragma unroll
                for (int k = 0; k < kConBatch; k++) {
                    const int r = r0 + k;
                    float strength = sv[k];
                    if (r < cnt && strength > 0) {
                        const bool isE = r < cntE;
                        if constexpr (Rng) {
                            if (P.condRng)
                                strength = near_failure(P, strength, isE, isE ? r : r - cntE, itype, condState, recNear,
                                                        nNearDraw);
                        }
                        if (strength > 0) {
                            if (isE) {
#pragma unroll
                                for (int ig = 0; ig < kMaxNG; ig++) {
                                    if (ig < ngE) {
                                        const float str = strength * ipE[ig];
                                        lgE[ig] += str * sm.og[ig][r];
                                        lhE[ig] += str * sm.oh[ig][r];
                                    }
                                }
                            } else {
#pragma unroll
                                for (int ig = 0; ig < kMaxNG; ig++) {
                                    if (ig < ngI) {
                                        const float str = strength * ipI[ig];
                                        lgI[ig] += str * sm.og[ig][r];
                                        lhI[ig] += str * sm.oh[ig][r];
                                    }
                                }
                            }
                        }
                    }
                }
            }
        }
        neuron_sync();
    }
    if (recNear) P.recNearCount[(size_t)(tp - P.recStep0) * nV1 + i] = nNearDraw;
    if (P.ffMode && P.ffMode != 3 && active && local < P.nE) {
        float *vAvg = P.ffPost + P.ffOffAvgE + 2 * (b * P.nE + local);
        learn_avg_delivery(P, __ldcg(sPrev + i), vAvg, vAvg + 1, vAvg);
    }
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        st.gE[ig] += lgE[ig]; st.hE[ig] += lhE[ig];
        st.gI[ig] += lgI[ig]; st.hI[ig] += lhI[ig];
    }
    // far sums of the failure path (already zero when no far presynaptic neuron spiked)
    if (P.farPullOn && active) {
#pragma unroll
        for (int q = 0; q < 2 * kMaxNG; q++) {
            if (q < ns) {
                const float fg = __ldcg(P.farPull + (size_t)(2 * q) * nV1 + i);
                const float fh = __ldcg(P.farPull + (size_t)(2 * q + 1) * nV1 + i);
#pragma unroll
                for (int ig = 0; ig < kMaxNG; ig++) {
                    if (q < ngE && ig == q) { st.gE[ig] += fg; st.hE[ig] += fh; }
                    if (q >= ngE && ig == q - ngE) { st.gI[ig] += fg; st.hI[ig] += fh; }
                }
            }
        }
    }
    // far events (sum_G adds them after the near delivery); the ring slot is cleared
    if (far) far_apply(P, farSlot, i, fin, st);
    if (P.rec && active) record_conductances(P, (int)(tp % P.recSlots), i, st);
}

// What a step reads of its neuron's type: the persistent kernels keep it in shared memory, as a few
// 16-byte reads in place of a dozen indexed reads of the kernel's parameters.
struct __align__(16) TypeConst {
    float4 level;      // vR, vThres, vT, tRef
    float4 membrane;   // gL, C, 1/C (div_pow2), tau_w
    float4 adex;       // deltaT, 1/deltaT (div_pow2), a, b
    float pFF[kMaxNG], pE[kMaxNG], pI[kMaxNG];
};

__device__ __forceinline__ TypeConst type_const(const V1Params &P, int itype) {
    TypeConst k;
    k.level = make_float4(P.vR[itype], P.vThres[itype], P.vT[itype], P.tRef[itype]);
    k.membrane = make_float4(P.gL[itype], P.C[itype], P.invC[itype], P.tau_w[itype]);
    k.adex = make_float4(P.deltaT[itype], P.invDeltaT[itype], P.a[itype], P.b[itype]);
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        k.pFF[ig] = ig < P.ngFF ? P.pFF[itype * P.ngFF + ig] : 0.f;
        k.pE[ig] = ig < P.ngE ? P.pE[itype * P.ngE + ig] : 0.f;
        k.pI[ig] = ig < P.ngI ? P.pI[itype * P.ngI + ig] : 0.f;
    }
    return k;
}

// The tonic drive of the AdEx constructor (src/coredynamics.cuh:41-49).
__device__ __forceinline__ float tonic_current(const V1Params &P, int itype, float tonic) {
    const float vT = P.vT[itype], gL = P.gL[itype], aa = P.a[itype], deltaT = P.deltaT[itype];
    const float targetV = P.vL + (vT - P.vL) * tonic;
    if (targetV > vT) return (gL + aa) * (targetV - P.vL) - gL * deltaT;
    return (gL + aa) * (targetV - P.vL) - gL * deltaT * expf((targetV - vT) / deltaT);
}

// One LGN synapse with spike word sFF and weight f (src/coredynamics.cu:1476-1500).
template <bool Rng>
__device__ __forceinline__ void lgn_input(const V1Params &P, const float *pFF, float sFF, float f, bool backingUp,
                                          float tBack, float pf, float nSynFF, float *g0, float *h0,
                                          float *g1, float *h1, curandStateMRG32k3a &condState,
                                          float *recFF, int &nFF) {
    const float dt = P.dt;
    const unsigned nspFF = (unsigned)floorf(sFF);
    if (nspFF == 0) return;
    const float tspFF = (sFF - nspFF) * dt;
    if constexpr (Rng) {
        if (pf > 0) {
            const float normed_std = sqrtf(pf * (1 - pf) / nSynFF);
            const float rnd = curand_normal(&condState);
            if (recFF) {
                if (nFF < P.recCap) recFF[nFF] = rnd;
                else atomicOr(P.err, kErrRecordOverflow);
            }
            nFF++;
            f *= 1 - pf + normed_std * rnd;
        }
    }
    if (f > 0) {
        const float ddt = backingUp ? tBack - tspFF : 0.f;
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < P.ngFF) {
                const float str = f * pFF[ig];
                if (backingUp && ddt > 0) cond_input(P.condFF, g0[ig], h0[ig], str * nspFF, ddt, ig);
                cond_input(P.condFF, g1[ig], h1[ig], str * nspFF, dt - tspFF, ig);
            }
        }
    }
}

// The LGN spikes of one step as a persistent thread knows them: which of its synapses received one,
// the first two spike words, ids ([group of four][kCta] from its column) and weights ([synapse][kCta]).
struct LgnIn {
    unsigned mask;
    float w0, w1;
    const int4 *ids;
    const float *wts;
};

__device__ __forceinline__ int synapse_id(const int4 *ids, int q);

// What the feed-forward half of a membrane step hands to the integration half.
struct FFStep {
    float g0[kMaxNG];          // feed-forward conductances at the start of the integrated interval
    float noise0, noise1, depOut;
};

// Phase B, first half: noise and the feed-forward conductances of step t (decay over the step and
// the LGN input, src/coredynamics.cu:1422-1502); st.gFF/hFF leave at their end-of-step values.
// Nothing here depends on what other neurons do in step t - 1, so the persistent kernels run it
// while they wait for them.  With SmemSyn the spikes are known (in); otherwise ids and words are
// loaded batch by batch and weights only for synapses that received a spike.
template <bool Rng, bool SmemSyn>
__device__ __forceinline__ void step_feedforward(const V1Params &P, const TypeConst &tc, long long t, int i, int itype,
                                                 float tonic, float depC, int m, const float *__restrict__ lgnSInfo, NState &st,
                                                 curandStateMRG32k3a &condState, curandStateMRG32k3a &noisyState,
                                                 FFStep &ff, const LgnIn &in = LgnIn{}) {
    const int nV1 = P.nV1;
    const float dt = P.dt;
    const int ngFF = P.ngFF;
    const float tBack = st.tBack;
    ff.noise0 = st.lastNoise;
    float h0[kMaxNG], g1[kMaxNG], h1[kMaxNG];
    float *g0 = ff.g0;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        g1[ig] = st.gFF[ig];
        h1[ig] = st.hFF[ig];
        g0[ig] = g1[ig];
        h0[ig] = h1[ig];
        if (ig < ngFF) cond_decay_step(P.condFF, P.decFF, g1[ig], h1[ig], ig);
    }
    // noise (src/coredynamics.cu:1422-1440)
    float noise1 = 0.f;
    if constexpr (Rng) {
        const float noiseRatio = P.noiseOnTonic ? tonic : 1.0f;
        noise1 = sqrtf(2 * P.noisyDep[itype] * (P.vT[itype] - P.vR[itype]) * noiseRatio * dt);
        if (noise1 > 0) {
            const float rnd = curand_normal(&noisyState);
            if (P.recNoise) {
                long long rs = t - P.recStep0;
                if (rs >= 0 && rs < P.recSteps) P.recNoise[(size_t)rs * nV1 + i] = rnd;
            }
            noise1 *= rnd;
            if (P.tau_noise > 0) {
                noise1 /= P.tau_noise;
                const float hk1 = -ff.noise0 / P.tau_noise;
                const float hk2 = -(ff.noise0 + dt * hk1 + noise1) / P.tau_noise;
                noise1 += ff.noise0 + dt * (hk1 + hk2) / 2;
                st.lastNoise = noise1;
            }
        }
    }
    ff.noise1 = noise1;
    const float pf = Rng ? P.synFailFF[itype] : 0.f;
    const float nSynFF = P.synPerConFF[itype];
    const bool backingUp = tBack < dt && tBack > 0;
    ff.depOut = depC + noise1;
    if (backingUp) {
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++)
            if (ig < ngFF) cond_decay(P.condFF, g0[ig], h0[ig], tBack, ig);
    }
    // LGN input (src/coredynamics.cu:1466-1502), synapse order kept
    float *recFF = nullptr;
    int nFF = 0;
    if (Rng && P.recFF) {
        long long rs = t - P.recStep0;
        if (rs >= 0 && rs < P.recSteps) recFF = P.recFF + ((size_t)rs * nV1 + i) * P.recCap;
    }
    if constexpr (SmemSyn) {
        // the synapses that received a spike, in synapse order; the first two words are here
        unsigned mask = in.mask;
        for (int k = 0; mask; k++) {
            const int q = __ffs(mask) - 1;
            mask &= mask - 1;
            const float sFF = k == 0 ? in.w0 : (k == 1 ? in.w1 : __ldcg(lgnSInfo + synapse_id(in.ids, q)));
            lgn_input<Rng>(P, tc.pFF, sFF, in.wts[q * kCta], backingUp, tBack, pf, nSynFF, g0, h0, g1, h1, condState,
                           recFF, nFF);
        }
    } else if (m <= kMaxLgnReg) {
        // ids and spike words in chunks of 16 (all loads of a chunk in flight together); the
        // weight is read only for synapses that received a spike, in synapse order
        unsigned mask = 0u;
#pragma unroll
        for (int c = 0; c < kMaxLgnReg; c += 16) {
            if (c < m) {
                int ids[16];
#pragma unroll
                for (int k = 0; k < 16; k++) ids[k] = c + k < m ? __ldg(P.lgnId + (size_t)(c + k) * nV1 + i) : 0;
#pragma unroll
                for (int k = 0; k < 16; k++)
                    mask |= ((c + k < m && __ldcg(lgnSInfo + ids[k]) >= 1.0f) ? 1u : 0u) << (c + k);
            }
        }
        while (mask) {
            const int q = __ffs(mask) - 1;
            mask &= mask - 1;
            const size_t lid = (size_t)q * nV1 + i;
            const float sFF = __ldcg(lgnSInfo + __ldg(P.lgnId + lid));
            const float f = __ldg(P.sLGN + lid);
            lgn_input<Rng>(P, tc.pFF, sFF, f, backingUp, tBack, pf, nSynFF, g0, h0, g1, h1, condState, recFF,
                           nFF);
        }
    } else {
        for (int q0 = 0; q0 < m; q0 += kLgnBatch) {
            int ids[kLgnBatch];
            float fs[kLgnBatch], sp[kLgnBatch];
#pragma unroll
            for (int k = 0; k < kLgnBatch; k++) {
                const size_t lid = (size_t)(q0 + k) * nV1 + i;
                ids[k] = q0 + k < m ? __ldg(P.lgnId + lid) : 0;
                fs[k] = q0 + k < m ? __ldg(P.sLGN + lid) : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kLgnBatch; k++) sp[k] = q0 + k < m ? __ldcg(lgnSInfo + ids[k]) : 0.f;
#pragma unroll
            for (int k = 0; k < kLgnBatch; k++) {
                if (q0 + k < m)
                    lgn_input<Rng>(P, tc.pFF, sp[k], fs[k], backingUp, tBack, pf, nSynFF, g0, h0, g1, h1, condState,
                                   recFF, nFF);
            }
        }
    }
    if (recFF) P.recFFCount[(size_t)(t - P.recStep0) * nV1 + i] = nFF;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        st.gFF[ig] = g1[ig];
        st.hFF[ig] = h1[ig];
    }
}

// Phase B, second half: cortical conductances, integration and threshold of step t
// (src/coredynamics.cu:1380-1590).  Returns the spike word.
__device__ __forceinline__ float step_membrane(const V1Params &P, const TypeConst &tc, float depC, const FFStep &ff,
                                               NState &st) {
    const float dt = P.dt;
    const int ngE = P.ngE, ngI = P.ngI, ngFF = P.ngFF;
    const float4 lvl = tc.level, mem = tc.membrane, adx = tc.adex;
    const float vR = lvl.x, vThres = lvl.y, vT = lvl.z, tRef = lvl.w;
    const float gL = mem.x, Cm = mem.y, invC = mem.z, tau_w = mem.w;
    const float deltaT = adx.x, invDeltaT = adx.y, aa = adx.z, bb = adx.w;
    const float v0 = st.v;
    float w0 = st.w;
    float tBack = st.tBack;
    const float noise0 = ff.noise0;
    float noise1 = ff.noise1;
    const bool backingUp = tBack < dt && tBack > 0;

    // cortical conductances: keep the start-of-step value, decay to the end
    float ge[kMaxNG], he[kMaxNG], gi[kMaxNG], hi[kMaxNG];
    float gE_t1 = 0.0f, gI_t1 = 0.0f;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        ge[ig] = st.gE[ig]; he[ig] = st.hE[ig];
        if (ig < ngE) {
            cond_decay_step(P.condE, P.decE, st.gE[ig], st.hE[ig], ig);
            gE_t1 += st.gE[ig];
        }
    }
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        gi[ig] = st.gI[ig]; hi[ig] = st.hI[ig];
        if (ig < ngI) {
            cond_decay_step(P.condI, P.decI, st.gI[ig], st.hI[ig], ig);
            gI_t1 += st.gI[ig];
        }
    }
    float gE_t0 = 0.0f;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ngFF) {
            gE_t0 += ff.g0[ig];
            gE_t1 += st.gFF[ig];
        }
    }
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ngE) {
            if (backingUp) cond_decay(P.condE, ge[ig], he[ig], tBack, ig);
            gE_t0 += ge[ig];
        }
    }
    float gI_t0 = 0.0f;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ngI) {
            if (backingUp) cond_decay(P.condI, gi[ig], hi[ig], tBack, ig);
            gI_t0 += gi[ig];
        }
    }
    // stepping (src/coredynamics.cu:1546-1590; AdEx src/coredynamics.cuh:27-118)
    float v = v0, w = w0, tsp = 0.f;
    int spikeCount = 0;
    if (tBack < dt) {
        const float a0 = gE_t0 + gI_t0 + gL;
        const float b0 = gE_t0 * P.vE + gI_t0 * P.vI + gL * P.vL + depC;
        const float a1 = gE_t1 + gI_t1 + gL;
        const float b1 = gE_t1 * P.vE + gI_t1 * P.vI + gL * P.vL + depC;
        const float new_dt = dt - tBack;
        if (backingUp) {
            const float A = aa * (v0 - P.vL);
            w0 = (w0 - A) * expf(-tBack / tau_w) + A;
        }
        float nz0, nz1;
        if (P.tau_noise > 0) { nz0 = noise0; nz1 = noise1; }
        else { noise1 = div_pow2(noise1, dt, P.invDt); nz0 = noise1; nz1 = noise1; }
        {
            const float dTgL = deltaT * gL;
            const float fk1 =
                div_pow2(-a0 * v0 + b0 + dTgL * expf(div_pow2(v0 - vT, deltaT, invDeltaT)) - w0, Cm, invC) + nz0;
            const float gk1 = div_sparse(aa * (v0 - P.vL) - w0, tau_w);
            const float v1 = v0 + new_dt * fk1;
            const float w1 = w0 + new_dt * gk1;
            const float fk2 =
                div_pow2(-a1 * v1 + b1 + dTgL * expf(div_pow2(v1 - vT, deltaT, invDeltaT)) - w1, Cm, invC) + nz1;
            const float gk2 = div_sparse(aa * (v1 - P.vL) - w1, tau_w);
            w = w0 + new_dt * (gk1 + gk2) / 2;
            v = v0 + new_dt * (fk1 + fk2) / 2;
        }
        if (v > vThres) {
            const float ratio = (vThres - v0) / (v - v0);
            tsp = tBack + ratio * new_dt;
            w0 += ratio * (w - w0) + bb;
            if (!(tsp >= 0)) atomicOr(P.err, kErrNegTsp);
            spikeCount = 1;
            tBack = tsp + tRef;
            v = vR;
        } else {
            if (tBack > 0) tBack = 0;
        }
    }
    if (tBack >= dt) {
        v = vR;
        const float A = aa * (v - P.vL);
        w = (w0 - A) * expf(-(dt - tsp) / tau_w) + A;
        tBack -= dt;
    }
    st.v = v;
    if (P.iModel == 1) st.w = w;
    st.tBack = tBack;
    return spikeCount > 0 ? 1.0f + tsp / dt : v;
}

// The step's spike word to global memory and to the records (ring slot recSlot).
__device__ __forceinline__ void store_step(const V1Params &P, long long t, int i, float sInfo, float depOut,
                                           const NState &st, int recSlot) {
    const int nV1 = P.nV1;
    __stcg(P.sInfo + (size_t)(t & 1) * nV1 + i, sInfo);
    if (P.recSpk) P.recSpk[(size_t)recSlot * nV1 + i] = sInfo;
    if (P.rec) {
        float *r = P.rec + recSlot * P.recStride;
        const RecOff o = rec_off(P);
        r[o.sinfo + i] = sInfo;
        r[o.dep + i] = depOut;
        if (P.iModel == 1) r[o.w + i] = st.w;
        r[o.v + i] = st.v;
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < P.ngFF) r[o.gFF + ig * nV1 + i] = st.gFF[ig];
            if (P.hWrite && ig < P.ngFF) r[o.hFF + ig * nV1 + i] = st.hFF[ig];
        }
    }
}

// Phase B: one membrane step of neuron i with its LGN synapses in global memory.
template <bool Rng>
__device__ __forceinline__ float step_neuron(const V1Params &P, long long t, int i, int itype, float tonic, float depC,
                                             int m, const float *__restrict__ lgnSInfo, NState &st,
                                             curandStateMRG32k3a &condState, curandStateMRG32k3a &noisyState) {
    FFStep ff;
    const TypeConst tc = type_const(P, itype);
    step_feedforward<Rng, false>(P, tc, t, i, itype, tonic, depC, m, lgnSInfo, st, condState, noisyState, ff);
    const float sInfo = step_membrane(P, tc, depC, ff, st);
    P.dep[i] = ff.depOut;
    store_step(P, t, i, sInfo, ff.depOut, st, P.recSpk || P.rec ? (int)(t % P.recSlots) : 0);
    return sInfo;
}

// Where a neuron's learning variables live: in global memory (per-step kernel), or in shared memory for the
// K steps of a launch (persistent kernel), with the synapses' weights and ids.
struct LearnVars {
    float *ltd, *trip, *avg0, *avg1;   // post traces; filtered rate (avg1: at the spike time, E with learning != 3)
    float *total, *target;             // total LGN weight and its target
    float *wts;                        // weights, wStride apart
    size_t wStride;
};

// Global places of neuron i's learning variables.
__device__ __forceinline__ LearnVars learn_vars(const V1Params &P, int i, int local) {
    const bool isE = local < P.nE;
    const int nEt = P.nE * P.nblock, nIt = P.nI * P.nblock, b = i / P.blockSize;
    const int id = isE ? b * P.nE + local : b * P.nI + (local - P.nE);   // eid / iid
    LearnVars v;
    v.ltd = (isE ? P.ffPost : P.ffPost + P.ffOffI) + id;
    v.trip = (isE ? P.ffPost + nEt : P.ffPost + P.ffOffI + nIt) + id;
    v.avg0 = isE ? P.ffPost + P.ffOffAvgE + 2 * id : P.ffPost + P.ffOffAvgI + id;
    v.avg1 = v.avg0 + 1;
    v.total = P.totalFF + i;
    v.target = P.totalFF + P.nV1 + i;
    v.wts = P.sLGNw + i;
    v.wStride = P.nV1;
    return v;
}

// Decay factors over a whole step of a type's post traces (the expressions learn_ff evaluates for other
// intervals).
struct LearnDecay {
    float ltd, trip, avg;
};
__device__ __forceinline__ LearnDecay learn_decay(const V1Params &P, const FFType &T) {
    return LearnDecay{expf(-P.dt / T.tauLTD), expf(-P.dt / T.tauTrip), expf(-P.dt / T.tauAvg)};
}

// LGN->V1 plasticity after the membrane step of neuron i (learning 1-3): the learning block
// of compute_V_collect_spike_learnFF_fast (src/coredynamics.cu:1631-1993) with one FF->E type
// for excitatory posts and, with learning 2, one FF->I type for inhibitory posts.  The post
// LTD and triplet traces and the filtered rate are read at the step start and, when the neuron
// spiked, decayed to its spike time tsp; each LGN synapse (in synapse order) takes the
// homeostatic factor, LTD when its LGN cell spiked (from the post LTD trace at the earlier of
// the two spike times, scaled by the squared filtered rate when targetFR > 0), LTP when the
// neuron spiked (the presynaptic trace at the step start or right after the LGN spike,
// whichever precedes tsp, decayed to tsp, times the post triplet trace), and is clipped to
// [gmin, gmax]; the post traces then take the spike count and decay to the end of the step.
// The reference's choices kept: with learning != 3 the excitatory filtered rate is not
// advanced here but stored at tsp into its second slot for the delivery to advance
// (vAvgE[2*eid+1], src/coredynamics.cu:1746-1748); the inhibitory posts' LTP reads
// presynaptic trace 0 (layer 1 + 3j of the LGN surface with j counting from 0,
// src/coredynamics.cu:1905-1912), which is the FF->E type's trace when both types learn.
// Float arithmetic in the reference's order.
//
// A warp's instructions bound it: every synapse of every lane in synapse order, with few warps per SM to
// hide the latency of each.  What a synapse whose cell did not spike shares with the others is computed once
// (the decay of its trace to tsp), and the words and traces of kLearnChunk synapses are read together (one
// by one, each waited for its own reads: 15 of the 26 us of a per-step launch).  In the persistent
// kernel (in: the step's LGN spikes; else null) only the words of cells that spiked are read, and weights, ids and the
// neuron's variables stay in shared memory for the K steps.  200 steps of 2 x 1,024 neurons with 20
// synapses: 6,221 us as launches per step, 2,359 us so (2,741 with each synapse's own expf and reads, 2,941
// with words and traces in registers for all ten synapses' paths: spills).
constexpr int kLearnChunk = 10;
constexpr int kLearnVars = 6;   // learning variables a persistent thread keeps in shared memory

__device__ __forceinline__ void learn_ff(const V1Params &P, int i, int local, int m, float sInfo,
                                         const float *__restrict__ lgnSInfo, const float *__restrict__ preRow, int nLGN,
                                         const LearnVars &v, const LearnDecay &decay, const LgnIn *in) {
    const bool isE = local < P.nE;
    if (!isE && !P.ffI) return;
    const FFType &T = P.ffT[isE ? 0 : 1];
    const float dt = P.dt;
    float nsp, tsp;
    if (sInfo > 0) {
        nsp = floorf(sInfo);
        tsp = (sInfo - nsp) * dt;
    } else {
        nsp = 0;
        tsp = dt;
    }
    // row 0: the step start; row 1: the spike time
    float lLTD[2], lTrip[2], lAvg[2];
    lLTD[0] = *v.ltd;
    lTrip[0] = *v.trip;
    lAvg[0] = *v.avg0;
    lLTD[1] = lTrip[1] = lAvg[1] = 0.f;
    if (nsp > 0) {
        lLTD[1] = lLTD[0];
        lTrip[1] = lTrip[0];
        lLTD[1] *= expf(-tsp / T.tauLTD);
        lTrip[1] *= expf(-tsp / T.tauTrip);
        lAvg[1] = lAvg[0];
        lAvg[1] *= expf(-tsp / T.tauAvg);
        if (isE && P.ffMode != 3) *v.avg1 = lAvg[1];
    }
    float new0 = 0.f, change = 0.f, delta_f = 0.f;
    if (P.applyHomeo) {
        const float f0 = *v.total;
        const float finf = *v.target;
        const float d = f0 - finf;
        if (d > 0 || P.symmetricHomeo) {
            new0 = d * P.expHomeo + finf;
            change = P.applyHomeo == 1 ? new0 / f0 : (new0 - f0) / (float)m;
        } else {
            new0 = f0;
            change = P.applyHomeo == 1 ? 1.f : 0.f;
        }
    }
    // the presynaptic trace decays over the same time for every LGN cell that did not spike before the neuron
    const float eLTP = nsp > 0 ? expf(-tsp / T.tauLTP) : 0.f;
    for (int q0 = 0; q0 < m; q0 += kLearnChunk) {
        float sFF[kLearnChunk], lpre[kLearnChunk];
        auto cell = [&](int q) { return in ? synapse_id(in->ids, q) : __ldg(P.lgnId + (size_t)q * P.nV1 + i); };
#pragma unroll
        for (int k = 0; k < kLearnChunk; k++) {
            const int q = q0 + k;
            sFF[k] = lpre[k] = 0.f;
            if (q < m && (!in || (in->mask >> q) & 1u)) sFF[k] = __ldcg(lgnSInfo + cell(q));
        }
        if (nsp > 0) {
#pragma unroll
            for (int k = 0; k < kLearnChunk; k++)
                if (q0 + k < m) lpre[k] = __ldcg(preRow + cell(q0 + k));
        }
#pragma unroll
        for (int k = 0; k < kLearnChunk; k++) {
            const int q = q0 + k;
            if (q >= m) break;
            float *w = v.wts + q * v.wStride;
            float f = *w;
            if (f == 0 && !P.rebound) continue;
            if (P.applyHomeo == 1) f *= change;
            else if (P.applyHomeo == 2) f += change;
            float pre = lpre[k], e = eLTP;
            if (sFF[k] > 0) {
                const float nspFF = floorf(sFF[k]);
                const float tspFF = (sFF[k] - nspFF) * dt;
                if (nspFF > 0) {  // LTD, whether or not the neuron spiked
                    const int cPick = tspFF < tsp ? 0 : 1;
                    const float delta_t = tspFF < tsp ? tspFF : tspFF - tsp;
                    float A_LTD = T.A_ratio;
                    if (T.targetFR > 0) A_LTD *= T.tauLTP * lAvg[cPick] * lAvg[cPick];
                    const float df = lLTD[cPick] * expf(-delta_t / T.tauLTD) * A_LTD;
                    f -= df;
                    if (P.applyHomeo) delta_f -= df;
                }
                if (nsp > 0 && tspFF < tsp) {
                    pre = __ldcg(preRow + nLGN + cell(q));
                    e = expf(-(tsp - tspFF) / T.tauLTP);
                }
            }
            if (nsp > 0) {  // LTP, whether or not the LGN cell spiked
                const float df = pre * e * lTrip[1] * T.A_LTP;
                if (P.applyHomeo) delta_f += df;
                f += df;
            }
            if (f < T.gmin) {
                if (P.applyHomeo) delta_f += T.gmin - f;
                f = T.gmin;
            }
            if (f > T.gmax) {
                if (P.applyHomeo) delta_f -= f - T.gmax;
                f = T.gmax;
            }
            *w = f;
        }
    }
    if (P.applyHomeo) *v.total = new0 + delta_f;
    // the post traces take this step's spikes and decay to its end
    const bool avg = !isE || P.ffMode == 3;
    if (nsp > 0) {
        const float delta_t = dt - tsp;
        *v.ltd = (lLTD[1] + nsp) * expf(-delta_t / T.tauLTD);
        *v.trip = (lTrip[1] + nsp) * expf(-delta_t / T.tauTrip);
        if (avg) *v.avg0 = (lAvg[1] + nsp) * expf(-delta_t / T.tauAvg);
    } else {
        *v.ltd = lLTD[0] * decay.ltd;
        *v.trip = lTrip[0] * decay.trip;
        if (avg) *v.avg0 = lAvg[0] * decay.avg;
    }
}

// Phase B when dt exceeds the shortest refractory period: a neuron may fire several times in
// one step (compute_V_collect_spike_learnFF, src/coredynamics.cu:427-845, without learning).
// After each spike whose refractory period ends inside the step the membrane is integrated
// again from the end of that period (tBack): the feed-forward and cortical conductances at
// tBack are advanced from the previous interval start, inputs arriving after the interval
// start and before tBack are added, w is carried with v held at vR, and RK2 runs over the rest
// of the step.  The end-of-step conductances (g1) and the failure draws come from the first
// pass only.  Kept from the reference: with tau_noise = 0 the noise term is divided by dt once
// more on every pass (src/coredynamics.cu:758-759).  The spike word is
// nsp + mean(tsp)/dt.  m <= kMaxLgnMulti (checked by the host).
template <bool Rng>
__device__ __noinline__ float step_neuron_multi(const V1Params &P, long long t, int i, int itype, float tonic, float depC,
                                   int m, const float *__restrict__ lgnSInfo, NState &st,
                                   curandStateMRG32k3a &condState, curandStateMRG32k3a &noisyState) {
    const int nV1 = P.nV1;
    const float dt = P.dt;
    const int ngE = P.ngE, ngI = P.ngI, ngFF = P.ngFF;
    const float vR = P.vR[itype], vThres = P.vThres[itype], gL = P.gL[itype];
    const float Cm = P.C[itype], tRef = P.tRef[itype], vT = P.vT[itype];
    const float deltaT = P.deltaT[itype], tau_w = P.tau_w[itype], aa = P.a[itype];
    const float bb = P.b[itype];
    float v0 = st.v;
    float w0 = st.w;
    float tBack = st.tBack;
    const float noise0 = st.lastNoise;
    float ge[kMaxNG], he[kMaxNG], gi[kMaxNG], hi[kMaxNG];
    float gE_t1 = 0.0f, gI_t1 = 0.0f;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        ge[ig] = st.gE[ig]; he[ig] = st.hE[ig];
        if (ig < ngE) {
            cond_decay_step(P.condE, P.decE, st.gE[ig], st.hE[ig], ig);
            gE_t1 += st.gE[ig];
        }
    }
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        gi[ig] = st.gI[ig]; hi[ig] = st.hI[ig];
        if (ig < ngI) {
            cond_decay_step(P.condI, P.decI, st.gI[ig], st.hI[ig], ig);
            gI_t1 += st.gI[ig];
        }
    }
    float g0[kMaxNG], h0[kMaxNG], g1[kMaxNG], h1[kMaxNG];
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        g1[ig] = st.gFF[ig];
        h1[ig] = st.hFF[ig];
        g0[ig] = g1[ig];
        h0[ig] = h1[ig];
        if (ig < ngFF) cond_decay_step(P.condFF, P.decFF, g1[ig], h1[ig], ig);
    }
    float noise1 = 0.f;
    if constexpr (Rng) {
        const float noiseRatio = P.noiseOnTonic ? tonic : 1.0f;
        noise1 = sqrtf(2 * P.noisyDep[itype] * (vT - vR) * noiseRatio * dt);
        if (noise1 > 0) {
            const float rnd = curand_normal(&noisyState);
            if (P.recNoise) {
                long long rs = t - P.recStep0;
                if (rs >= 0 && rs < P.recSteps) P.recNoise[(size_t)rs * nV1 + i] = rnd;
            }
            noise1 *= rnd;
            if (P.tau_noise > 0) {
                noise1 /= P.tau_noise;
                const float hk1 = -noise0 / P.tau_noise;
                const float hk2 = -(noise0 + dt * hk1 + noise1) / P.tau_noise;
                noise1 += noise0 + dt * (hk1 + hk2) / 2;
                st.lastNoise = noise1;
            }
        }
    }
    const float pf = Rng ? P.synFailFF[itype] : 0.f;
    const float nSynFF = P.synPerConFF[itype];
    const float depOut = depC + noise1;
    P.dep[i] = depOut;
    float *recFF = nullptr;
    int nFF = 0;
    if (Rng && P.recFF) {
        long long rs = t - P.recStep0;
        if (rs >= 0 && rs < P.recSteps) recFF = P.recFF + ((size_t)rs * nV1 + i) * P.recCap;
    }
    float fmod[kMaxLgnMulti];
    const int mm = m < kMaxLgnMulti ? m : kMaxLgnMulti;
    bool backingUp = tBack < dt && tBack > 0;
    float new_t0 = 0.f, tspSum = 0.f, v = v0, w = w0, tsp = 0.f;
    float a1 = 0.f, b1 = 0.f;
    int spikeCount = 0, pass = 0;
    do {
        const float dtBack = backingUp ? tBack - new_t0 : 0.f;
        if (backingUp) {
#pragma unroll
            for (int ig = 0; ig < kMaxNG; ig++)
                if (ig < ngFF) cond_decay(P.condFF, g0[ig], h0[ig], dtBack, ig);
        }
        for (int q = 0; q < mm; q++) {
            const size_t lid = (size_t)q * nV1 + i;
            if (spikeCount == 0) fmod[q] = __ldg(P.sLGN + lid);
            const float sFF = __ldcg(lgnSInfo + __ldg(P.lgnId + lid));
            const unsigned nspFF = (unsigned)floorf(sFF);
            const float tspFF = (sFF - nspFF) * dt;
            if (nspFF > 0 && tspFF >= new_t0) {
                if constexpr (Rng) {
                    if (spikeCount == 0 && pf > 0) {
                        const float normed_std = sqrtf(pf * (1 - pf) / nSynFF);
                        const float rnd = curand_normal(&condState);
                        if (recFF) {
                            if (nFF < P.recCap) recFF[nFF] = rnd;
                            else atomicOr(P.err, kErrRecordOverflow);
                        }
                        nFF++;
                        fmod[q] *= 1 - pf + normed_std * rnd;
                    }
                }
                if (fmod[q] > 0) {
                    const float ddt = backingUp ? tBack - tspFF : 0.f;
#pragma unroll
                    for (int ig = 0; ig < kMaxNG; ig++) {
                        if (ig < ngFF) {
                            const float str = fmod[q] * P.pFF[itype * ngFF + ig];
                            if (backingUp && ddt > 0) cond_input(P.condFF, g0[ig], h0[ig], str * nspFF, ddt, ig);
                            if (spikeCount == 0) cond_input(P.condFF, g1[ig], h1[ig], str * nspFF, dt - tspFF, ig);
                        }
                    }
                }
            }
        }
        float gE_t0 = 0.0f;
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < ngFF) {
                gE_t0 += g0[ig];
                if (spikeCount == 0) gE_t1 += g1[ig];
            }
        }
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < ngE) {
                if (backingUp) cond_decay(P.condE, ge[ig], he[ig], dtBack, ig);
                gE_t0 += ge[ig];
            }
        }
        float gI_t0 = 0.0f;
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < ngI) {
                if (backingUp) cond_decay(P.condI, gi[ig], hi[ig], dtBack, ig);
                gI_t0 += gi[ig];
            }
        }
        tsp = 0.f;
        if (tBack < dt) {
            const float a0 = gE_t0 + gI_t0 + gL;
            const float b0 = gE_t0 * P.vE + gI_t0 * P.vI + gL * P.vL + depC;
            if (spikeCount == 0) {
                a1 = gE_t1 + gI_t1 + gL;
                b1 = gE_t1 * P.vE + gI_t1 * P.vI + gL * P.vL + depC;
            }
            const float new_dt = dt - tBack;
            if (backingUp) {
                const float A = aa * (v0 - P.vL);
                w0 = (w0 - A) * expf(-dtBack / tau_w) + A;
            }
            float nz0, nz1;
            if (P.tau_noise > 0) { nz0 = noise0; nz1 = noise1; }
            else { noise1 /= dt; nz0 = noise1; nz1 = noise1; }
            const float dTgL = deltaT * gL;
            const float fk1 = (-a0 * v0 + b0 + dTgL * expf((v0 - vT) / deltaT) - w0) / Cm + nz0;
            const float gk1 = (aa * (v0 - P.vL) - w0) / tau_w;
            const float v1 = v0 + new_dt * fk1;
            const float w1 = w0 + new_dt * gk1;
            const float fk2 = (-a1 * v1 + b1 + dTgL * expf((v1 - vT) / deltaT) - w1) / Cm + nz1;
            const float gk2 = (aa * (v1 - P.vL) - w1) / tau_w;
            w = w0 + new_dt * (gk1 + gk2) / 2;
            v = v0 + new_dt * (fk1 + fk2) / 2;
            if (v > vThres) {
                new_t0 = tBack;
                const float ratio = (vThres - v0) / (v - v0);
                tsp = new_t0 + ratio * new_dt;
                w0 += ratio * (w - w0) + bb;
                if (!(tsp >= 0)) atomicOr(P.err, kErrNegTsp);
                tspSum += tsp;
                spikeCount++;
                tBack = tsp + tRef;
                backingUp = tBack < dt;
                if (backingUp) v0 = vR;
                else v = vR;
            } else {
                if (tBack > 0) tBack = 0;
                backingUp = false;
            }
        }
        if (tBack >= dt) {
            v = vR;
            const float A = aa * (v - P.vL);
            w = (w0 - A) * expf(-(dt - tsp) / tau_w) + A;
            tBack -= dt;
        }
        if (++pass >= kMaxSpikePasses && backingUp) {
            atomicOr(P.err, kErrBounds);   // more passes than the refractory periods allow
            break;
        }
    } while (backingUp);
    if (recFF) P.recFFCount[(size_t)(t - P.recStep0) * nV1 + i] = nFF;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        st.gFF[ig] = g1[ig];
        st.hFF[ig] = h1[ig];
    }
    const float sInfo = spikeCount > 0 ? tspSum / (spikeCount * dt) + spikeCount : v;
    st.v = v;
    if (P.iModel == 1) st.w = w;
    st.tBack = tBack;
    __stcg(P.sInfo + (size_t)(t & 1) * nV1 + i, sInfo);
    if (P.recSpk) P.recSpk[(size_t)(t % P.recSlots) * nV1 + i] = sInfo;
    if (P.rec) {
        const long long slot = t % P.recSlots;
        float *r = P.rec + slot * P.recStride;
        const RecOff o = rec_off(P);
        r[o.sinfo + i] = sInfo;
        r[o.dep + i] = depOut;
        if (P.iModel == 1) r[o.w + i] = w;
        r[o.v + i] = v;
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (ig < ngFF) r[o.gFF + ig * nV1 + i] = g1[ig];
            if (P.hWrite && ig < ngFF) r[o.hFF + ig * nV1 + i] = h1[ig];
        }
    }
    return sInfo;
}

// step_neuron_multi on copies of the state: passing the caller's own by reference to a function
// that is not inlined would keep them in local memory for the whole kernel.
template <bool Rng>
__device__ __forceinline__ float step_multi(const V1Params &P, long long t, int i, int itype, float tonic, float depC, int m,
                                            const float *__restrict__ lgnSInfo, NState &st,
                                            curandStateMRG32k3a &condState, curandStateMRG32k3a &noisyState) {
    NState s = st;
    curandStateMRG32k3a a, b;
    if (Rng) {
        a = condState;
        b = noisyState;
    }
    const float sInfo = step_neuron_multi<Rng>(P, t, i, itype, tonic, depC, m, lgnSInfo, s, a, b);
    st = s;
    if (Rng) {
        condState = a;
        noisyState = b;
    }
    return sInfo;
}

// One delayed event: the spike of a neuron at step t (spike word sI, excitatory: preE) through
// a delayed synapse, in its k-th arrival slot; arrival step and offset as recal_G_vec
// (src/coredynamics.cu:282-333) and recal_G_mat (2163-2200) compute them, with explicitly
// rounded operations.  `code` is the synapse's packed word: whole-step delay in bits 0-15, post
// type in bits 16-23, class in bit 24 (1: near block, delivered through nearAcc; 0: far, through
// farAcc).  Offset of the event in its arrival step; the event exists if 0 <= offset < dt.
__device__ __forceinline__ float far_offset(const V1Params &P, float sI, float frac, int kk) {
    // dtsp = (sInfo - nsp + k)*dt - time2post, rounded step by step
    const float x = __fadd_rn(__fsub_rn(sI, (float)(unsigned)floorf(sI)), (float)kk);
    return __fsub_rn(__fmul_rn(x, P.dt), frac);
}

__device__ __forceinline__ void far_add(const V1Params &P, long long t, int tSlot, bool preE, float sI, int post,
                                        float f, int code, float dtsp, int kk) {
    const int ptype = (code >> 16) & 0xff;
    const bool nearClass = (code >> 24) & 1;
    const int ahead = (code & 0xffff) - kk;   // arrival step - t
    const unsigned nsp = (unsigned)floorf(sI);
    if (ahead < 0 || ahead >= P.farDepth - 1) {
        atomicOr(P.err, kErrFarOverflow);
        return;
    }
    const int nV1 = P.nV1;
    const int ns = P.ngE + P.ngI;
    const int ng = preE ? P.ngE : P.ngI;
    const int qoff = preE ? 0 : P.ngE;
    const float delta = __fsub_rn(P.dt, dtsp);
    // ring slot of the arrival step: tSlot is step t's (t mod farDepth, in [0, farDepth)) and 0 <=
    // ahead < farDepth - 1 (the only arrival before step 0 is the delivery that precedes the first
    // step when there are initial spikes: step -1, slot farDepth - 1)
    int aSlot = tSlot + ahead;
    if (aSlot >= P.farDepth) aSlot -= P.farDepth;
    unsigned long long *acc = (nearClass ? P.nearAcc : P.farAcc) + (size_t)aSlot * ns * 2 * nV1;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ng) {
            const float ip = preE ? P.pE[ptype * P.ngE + ig] : P.pI[ptype * P.ngI + ig];
            const float fv = __fmul_rn(__fmul_rn((float)nsp, f), ip);
            // conductance input of the arrival (cond_input of src/condShape.h:42-51) with the
            // hardware exponential and division (within a few ulp): the reference computes far
            // arrivals on the host, so no device expression reproduces its bits, and the
            // fixed-point ring already sums delayed near events in another order than its
            // recal_G_mat; the precise forms cost 14% of the step here
            const float rise = preE ? P.condE.rise[ig] : P.condI.rise[ig];
            const float dec = preE ? P.condE.decay[ig] : P.condI.decay[ig];
            const float dod = preE ? P.condE.dod[ig] : P.condI.dod[ig];
            const float etr = __expf(-__fdividef(delta, rise));
            const float g = fv * dod * (__expf(-__fdividef(delta, dec)) - etr);
            const float h = fv * etr;
            atomicAdd(&acc[(size_t)(2 * (qoff + ig)) * nV1 + post], (unsigned long long)far_to_fixed(g));
            atomicAdd(&acc[(size_t)(2 * (qoff + ig) + 1) * nV1 + post], (unsigned long long)far_to_fixed(h));
        }
    }
}

__device__ __forceinline__ void far_event(const V1Params &P, long long t, int tSlot, int pre, float sI, int post,
                                          float f, int code, float frac, int kk) {
    const float dtsp = far_offset(P, sI, frac, kk);
    if (dtsp < P.dt && dtsp >= 0 && f > 0)
        far_add(P, t, tSlot, (pre % P.blockSize) < P.nE, sI, post, f, code, dtsp, kk);
}

// Pushes the delayed events of up to 32 spikers of step t, one per lane (e0: first synapse, deg:
// synapses, sI: spike word, preE; lanes without one: deg 0), with all lanes of the warps that
// share them: warp `part` of `parts`.  sameStep: the events arriving in step t itself (whole-step
// delay 0 or 1 with as many whole steps of the window, deg then counts only such synapses);
// otherwise those arriving later.  A lane's items are 32 * parts apart; U of them are fetched
// together.  The fixed-point ring makes the sums independent of who pushes what, and in which
// order.
template <int U>
__device__ __forceinline__ void push_spikers(const V1Params &P, long long t, int tSlot, int e0, int deg, float sI,
                                             bool preE, bool sameStep, int part, int parts) {
    const int lane = threadIdx.x & 31;
    int incl = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    // synapse of item w of the owning lane r: e0[r] + w - (incl[r] - deg[r])
    const int shift = e0 - (incl - deg);
    const unsigned packed = __ballot_sync(0xffffffffu, preE);
    const float dt = P.dt;
    for (int base = part * 32; base < total; base += U * parts * 32) {
        int4 rc[U];
        int own[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int w = base + u * parts * 32 + lane;
            // first lane whose inclusive count exceeds w
            int lo = 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int y = __shfl_sync(0xffffffffu, incl, lo + o - 1);
                if (y <= w) lo += o;
            }
            const int e = __shfl_sync(0xffffffffu, shift, lo & 31) + w;
            own[u] = w < total ? lo : -1;
            if (w < total) rc[u] = __ldg(P.farRec + e);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const float s = __shfl_sync(0xffffffffu, sI, own[u] & 31);
            if (own[u] < 0) continue;
            const bool pe = (packed >> own[u]) & 1;
            const float f = __int_as_float(rc[u].y), frac = __int_as_float(rc[u].w);
            const int code = rc[u].z, steps = code & 0xffff;
            // the two arrival slots of the spike; at most one holds the event, up to rounding
            const float d0 = far_offset(P, s, frac, 0), d1 = far_offset(P, s, frac, 1);
            const bool k0 = d0 < dt && d0 >= 0 && f > 0 && (steps == 0) == sameStep;
            const bool k1 = d1 < dt && d1 >= 0 && f > 0 && (steps == 1) == sameStep;
            if (k0 || k1) far_add(P, t, tSlot, pe, s, rc[u].x, f, code, k0 ? d0 : d1, k0 ? 0 : 1);
            if (k0 && k1) far_add(P, t, tSlot, pe, s, rc[u].x, f, code, d1, 1);
        }
    }
}

// Spiker count (high 32 bits) and synapse work (low 32 bits) of step tl's far list.
__device__ __forceinline__ unsigned long long far_list_size(const V1Params &P, long long tl) {
    return __ldcg(P.farCount + (int)((tl + 3) % 3));
}

// The far events of step tl's spikes that arrive after step tl, from the step's global spiker list
// (the per-step kernels push them in step tl + 1), shared by the kCta-thread groups of nCta CTAs.
__device__ __forceinline__ void far_push_list(const V1Params &P, long long tl, int cta, int nCta) {
    const int n = (int)(far_list_size(P, tl) >> 32);
    if (n == 0) return;
    const int4 *list = P.farList + (size_t)((tl + 3) % 3) * P.nV1;  // tl >= -1
    const int tSlot = far_ring_slot(P, tl);
    const int lane = threadIdx.x & 31;
    for (int c0 = 0; c0 < n; c0 += 32) {
        int4 e = make_int4(0, 0, 0, 0);
        if (c0 + lane < n) e = __ldcg(list + c0 + lane);
        push_spikers<2>(P, tl, tSlot, e.y, e.z, __int_as_float(e.w), (e.x % P.blockSize) < P.nE, false,
                        cta * kWarps + (threadIdx.x >> 5), nCta * kWarps);
    }
}

// The far events of step t that arrive within step t itself (whole-step delay 0 or 1: the first n1
// synapses of each list), which must be in the ring before the next step delivers it: each
// warp pushes its own spikers'.  Also raises step t's flag of far presynaptic spikes and
// clears the next step's (its last readers are two steps back).
__device__ __forceinline__ void far_same_step(const V1Params &P, long long t, int t3, int tSlot, bool spk, float sInfo,
                                              bool isFarPre, bool preE, int e0, int n1, bool first) {
    if (first) P.farFlag[t3 == 2 ? 0 : t3 + 1] = 0;
    if (spk && sInfo > 1.0f && isFarPre) P.farFlag[t3] = 1;
    if (__any_sync(0xffffffffu, spk && n1 > 0))
        push_spikers<1>(P, t, tSlot, e0, spk ? n1 : 0, sInfo, preE, true, 0, 1);
}

// Phase C of the per-step kernels (runs in step t): appends this CTA's far presynaptic spikers to
// step t's global list (one atomic per warp) and pushes their same-step events.
__device__ __forceinline__ void far_phase(const V1Params &P, long long t, int i, bool active, float sInfo,
                                          bool isFarPre, bool preE, int e0, int deg, int n1, int cta) {
    const int t3 = (int)(t % 3);
    const bool first = cta == 0 && threadIdx.x == 0;
    if (first) P.farCount[(t + 1) % 3] = 0ull;
    const bool spk = active && sInfo >= 1.0f;
    const int lane = threadIdx.x & 31;
    const bool app = spk && deg > 0;
    const unsigned ab = __ballot_sync(0xffffffffu, app);
    if (ab) {
        const int leader = __ffs(ab) - 1;
        // one atomic per warp adds its spikers (high half) and their synapses (low half)
        const unsigned wsum = __reduce_add_sync(0xffffffffu, app ? (unsigned)deg : 0u);
        int base = 0;
        if (lane == leader)
            base = (int)(atomicAdd(P.farCount + t3, ((unsigned long long)__popc(ab) << 32) | wsum) >> 32);
        base = __shfl_sync(0xffffffffu, base, leader);
        if (app)
            P.farList[(size_t)t3 * P.nV1 + base + __popc(ab & ((1u << lane) - 1u))] =
                make_int4(i, e0, deg, __float_as_int(sInfo));
    }
    far_same_step(P, t, t3, far_ring_slot(P, t), spk, sInfo, isFarPre, preE, e0, n1, first);
}

// One V1 step (with the delivery of the previous step first) for CTA `cta` of the nCta CTAs
// that hold one patch: the per-step kernel and the batched kernel run this body.
template <bool Rng>
__device__ __forceinline__ void v1_step_body(const V1Params &P, long long t, int cta, int nCta,
                                             const float *__restrict__ lgnRing, int lgnSlots,
                                             int deliverPrev, int doStep, Smem &sm) {
    const int bs = P.blockSize;
    const int nq = (bs + kCta - 1) / kCta;
    const int b = cta / nq;
    const int local = (cta % nq) * kCta + threadIdx.x;
    const bool active = local < bs;
    const int i = b * bs + (active ? local : 0);
    const int itype = type_of(P, active ? local : 0);

    NState st;
    load_state(P, i, st);
    curandStateMRG32k3a condState, noisyState;
    if (Rng && P.condRng && active) condState = P.rGenCond[i];
    if (Rng && P.noiseRng && active) noisyState = P.rNoisy[i];

    if (deliverPrev) deliver_prev<Rng>(P, t - 1, b, local, i, active, itype, st, condState, sm);
    if (!doStep) {
        if (active) {
            store_state(P, i, st);
            if (Rng && P.condRng) P.rGenCond[i] = condState;
        }
        return;
    }
    float sInfo = 0.f;
    if (active) {
        const float tonic = P.tonicDep[i];
        const float depC = tonic_current(P, itype, tonic);
        const float *lgnSInfo = lgnRing + (size_t)(t % lgnSlots) * P.lgnN;
        if (P.multiSpike)
            sInfo = step_multi<Rng>(P, t, i, itype, tonic, depC, P.nLGNperV1[i], lgnSInfo, st, condState, noisyState);
        else
            sInfo = step_neuron<Rng>(P, t, i, itype, tonic, depC, P.nLGNperV1[i], lgnSInfo, st, condState, noisyState);
        store_state(P, i, st);
        if (Rng && P.condRng) P.rGenCond[i] = condState;
        if (Rng && P.noiseRng) P.rNoisy[i] = noisyState;
        if (P.spikeCount && sInfo >= 1.0f) P.spikeCount[i] += (unsigned)floorf(sInfo);
        if (P.farPullOn || P.nearPullOn) P.sRing[(size_t)(t % P.sDepth) * P.nV1 + i] = sInfo;
        if (P.ffLearn)
            learn_ff(P, i, local, P.nLGNperV1[i], sInfo, lgnSInfo,
                     P.ffPreRing + (size_t)(t % lgnSlots) * P.ffTypes * 2 * P.lgnN, P.lgnN, learn_vars(P, i, local),
                     learn_decay(P, P.ffT[local < P.nE ? 0 : 1]), nullptr);
    }
    if (P.farOn) {
        const int e0 = active ? P.farOff[i] : 0;
        const int deg = active ? P.farOff[i + 1] - e0 : 0;
        const int n1 = active ? P.farN1[i] : 0;
        const bool isFarPre = active && P.farPre[i];
        far_push_list(P, t - 1, cta, nCta);
        far_phase(P, t, i, active, sInfo, isFarPre, local < P.nE, e0, deg, n1, cta);
    }
}

template <bool Rng>
__global__ void __launch_bounds__(kCta) v1_step_kernel(V1Params P, const long long *stepBase,
                                                       int stepOffset,
                                                       const float *__restrict__ lgnRing,
                                                       int lgnSlots, int deliverPrev,
                                                       int doStep) {
    __shared__ Smem sm;
    const long long t = *stepBase + stepOffset;
    v1_step_body<Rng>(P, t, blockIdx.x, gridDim.x, lgnRing, lgnSlots, deliverPrev, doStep, sm);
}

// ---- K steps in one launch (persistent kernels) ----
// What a step of a patch waits for, and how the kernels below keep it short:
//   * the spikes of its own block (near delivery).  The CTAs of a block form a cluster: a thread
//     that spikes writes its unit conductances into the shared memory of every CTA of the block and
//     each warp its ballot word, as asynchronous stores that count towards an mbarrier there; a
//     step's phase completes when every warp of the block has announced its bytes and they have
//     landed.  No fence and no CTA barrier: every warp walks the block's ballot words itself.
//     Two buffers (parity of the step): a warp writes step t + 1's only after the phase of step
//     t, in which its peers announced that they had read step t - 1's.
//   * the far events arriving in the step, in the global ring.  A grid barrier per step orders the
//     same-step pushes before their delivery; a block without far synapses or foreign
//     neighbours needs none (one barrier per launch, after its first step, still bounds the
//     start of the grid).  Between its arrival and its wait a CTA does everything of the next step
//     that does not depend on other blocks: the near delivery and the feed-forward conductances.
//   * the LGN spikes: one bit per cell, a row per step copied to shared memory a step ahead by the
//     bulk-copy engine; a neuron tests the bits of its synapses and reads the words of those that
//     spiked (the words of all of them, 20 scattered copies per thread and step, took 1,850 cycles
//     of an 11,000-cycle step).
//   * the far pushes.  The CTA's spikers are listed in shared memory for kCta further threads of the
//     CTA (push warps): they push the same-step events, arrive at the grid barrier and then push the later
//     events, while the neuron threads are in the next step (waiting for their own pushes and the
//     release behind them, the neuron threads lost 2,300 of an 18,600-cycle step of 32 blocks).  Where the registers do
//     not allow the extra warps (two CTAs per SM) the neuron threads push themselves, between arrival and
//     wait.
// Bound by the latency of one warp's instruction stream (two warps per scheduler).  Measured per
// call, against general CTAs with a full grid barrier per step and LGN words per synapse: one block
// 800 steps 5,698 -> 3,492 us, 4 blocks with noise and failures 301 steps 3,128 -> 2,025, 8 blocks
// with far synapses 203 steps 2,260 -> 1,689, the 32-block patch with its movie 800 steps 13,039 ->
// 10,737; 12 trials of 4 blocks in one sweep 29,617 -> 16,424.
constexpr unsigned kBarrierAbort = 0x80000000u;
constexpr int kPushU = 2;       // far items a lane fetches together
constexpr int kMaxBitWords = 2048;   // LGN spike bits kept in shared memory (two rows of up to 65,536 cells)
// Polls of an mbarrier before it counts as lost.  A poll suspends its warp for up to 3.9 us, one of the grid
// barrier takes about 50 ns: a wait for other CTAs gets one for kGridPolls of the plan's limit, a
// wait for the CTA's own warps and copies a second.
constexpr int kMbarSpins = 1 << 18;
constexpr int kGridPolls = 64;

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned smem_at(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned at_rank(unsigned addr, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void send_word(unsigned addr, unsigned bar, unsigned v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send_float4(unsigned addr, unsigned bar, float4 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)),
                 "r"(__float_as_uint(v.w)), "r"(bar)
                 : "memory");
}
// One arrival at a peer's mbarrier that announces `bytes` of asynchronous stores.
__device__ __forceinline__ void announce(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// One poll of a phase.
__device__ __forceinline__ unsigned mbar_poll(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// Bounded wait of a whole warp for a phase; false (for all its lanes) if it does not complete, or, with
// stop, once a warp of the block has given up.
__device__ __noinline__ bool mbar_wait(unsigned bar, unsigned parity, int spins, const int *stop) {
    unsigned ok = mbar_poll(bar, parity);
    for (int i = 0; i < spins && !ok; i++) {
        if (stop && *(volatile const int *)stop) break;
        ok = mbar_poll(bar, parity);
    }
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void store_remote(unsigned addr, unsigned v) {
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Shared memory of a persistent CTA.
struct __align__(16) PShared {
    union {
        struct {
            float4 unit[2][kMaxBS];         // g, h per species of the block's spikers, by parity of the step
            unsigned ball[2][kMaxBS / 32];  // who spiked
        } list;
        Smem near;                          // general neighbour lists
    };
    uint64_t nearBar[2], bitBar[2];
    TypeConst type[kMaxType];
    // this CTA's far spikers, by parity of the step
    int cnt[2];
    int e0[2][kCta], deg[2][kCta], n1[2][kCta];
    float si[2][kCta];
    unsigned char preE[2][kCta];
    int stop;                       // a warp of the block gave up: the waits for spikes end
    unsigned left[kMaxBS / 32];     // leave_block: the block's warps
    int abortStep;
};
static_assert(kMaxNG == 2, "a spiker's unit conductances are two (g, h) pairs");

// Phases of the mbarriers (bit k: the parity the next wait on that barrier expects); they run on over
// the trials of a batch.
struct Phases {
    unsigned near0 = 0, near1 = 0, bit0 = 0, bit1 = 0;
};

// Sets up the mbarriers, once per launch; every thread of the CTA (and of its cluster) calls it.
__device__ __forceinline__ void init_barriers(PShared &sm, int csize) {
    if (threadIdx.x == 0) {
        for (int k = 0; k < 2; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_at(&sm.nearBar[k])), "r"(csize * kWarps));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_at(&sm.bitBar[k])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// Giving up.  A wait that runs out must not leave anyone waiting for good, nor end a CTA to which others
// still send.  So a warp whose wait for spikes or bits ran out (lost) tells all who may wait for it
// (give_up) and leaves where its CTA can tell that it does: at the next meeting of the CTA's warps, if
// there is one (a warp must not miss a barrier of a fixed number of threads), else where it is.  A step's
// meeting is behind its wait for the grid, and for all warps alike.  At the end the warps of a block
// tell each other how far they came; if one gave up they make up the announcements that are missing
// and stay until what they were sent has arrived (leave_block).
__device__ __noinline__ void give_up(PShared &sm, int csize, int *err, unsigned *count) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        atomicOr(err, kErrBarrier);
        if (count) atomicOr(count, kBarrierAbort);
    }
    if (csize == 1) *(volatile int *)&sm.stop = 1;
    else if (lane < csize) store_remote(at_rank(smem_at(&sm.stop), lane), 1u);
}

// Grid (or trial) barrier: two monotonic arrival counters, zeroed before each launch: the ends of the
// CTAs' steps, and the CTAs that have started.  meet: the neuron threads of a CTA meet, after one
// counter (if given) has reached its target.  False for all of them if a warp is lost, if that
// takes more than `limit` polls (sets kErrBarrier and the abort bit of the counter, which releases
// and fails every other waiter) or if the abort bit is set.
__device__ __forceinline__ bool meet(unsigned *count, unsigned target, bool lost, int *err, long long limit) {
    if (count && threadIdx.x == 0 && !lost) {
        unsigned c = 0;
        long long spins = 0;
        while (true) {
            if (++spins > limit) {
                atomicOr(err, kErrBarrier);
                atomicOr(count, kBarrierAbort);
                c = kBarrierAbort;
                break;
            }
            if (spins > 64) __nanosleep(32);
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
            if ((c & ~kBarrierAbort) >= target || (c & kBarrierAbort)) break;
        }
        lost = (c & kBarrierAbort) != 0;
    }
    __syncwarp();
    unsigned any;
    asm volatile("{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.or.pred q, 1, %2, p; selp.u32 %0, 1, 0, q; }"
                 : "=r"(any)
                 : "r"((unsigned)lost), "n"(kCta)
                 : "memory");
    return any == 0;
}

// This step's spikes of the warp (CTA `rank` of the block's csize) to every CTA of the block: unit
// conductances (output_g/h of compute_V, src/coredynamics.cu:2008-2041) and the ballot word.
__device__ __forceinline__ void publish_spikes(const V1Params &P, PShared &sm, int par, int csize, int rank, bool spk,
                                               float sInfo, bool isE) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, spk);
    const unsigned bar = smem_at(&sm.nearBar[par]);
    if (spk) {
        const float nsp = floorf(sInfo);
        const float tsp = (sInfo - nsp) * P.dt;
        float g[kMaxNG] = {0.f, 0.f}, h[kMaxNG] = {0.f, 0.f};
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            if (isE) {
                if (ig < P.ngE) cond_input(P.condE, g[ig], h[ig], nsp, P.dt - tsp, ig);
            } else {
                if (ig < P.ngI) cond_input(P.condI, g[ig], h[ig], nsp, P.dt - tsp, ig);
            }
        }
        const float4 u = make_float4(g[0], h[0], g[1], h[1]);
        if (csize == 1) {
            sm.list.unit[par][threadIdx.x] = u;
        } else {
            const unsigned to = smem_at(&sm.list.unit[par][rank * kCta + threadIdx.x]);
            for (int r = 0; r < csize; r++) send_float4(at_rank(to, r), at_rank(bar, r), u);
        }
    }
    if (csize == 1) {   // a block of one CTA is no cluster: plain stores and a plain arrival
        __syncwarp();
        if (lane == 0) {
            sm.list.ball[par][warp] = bal;
            asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
        }
    } else if (lane < csize) {
        const unsigned peer = at_rank(bar, lane);
        send_word(at_rank(smem_at(&sm.list.ball[par][rank * kWarps + warp]), lane), peer, bal);
        announce(peer, 4u + 16u * __popc(bal));
    }
}

// The end of a block's steps, for all threads of its csize CTAs (a cluster if exchange, with the spikes
// sent between them).  sent: the first step from t0 whose spikes this warp did not publish, due: the first
// one whose spikes it did not take.  False for all of them if one of them failed.  The warps of a block
// are at most a step apart in what they published, so that what is made up goes to the phases the
// peers still wait for.
__device__ __noinline__ bool leave_block(PShared &sm, bool exchange, int csize, int rank, long long t0, int sent, int due,
                                         bool failed, Phases ph) {
    if (!exchange || csize == 1) return __syncthreads_or(failed) == 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < kWarps && lane < csize)
        store_remote(at_rank(smem_at(&sm.left[rank * kWarps + warp]), lane), (unsigned)sent | (failed ? 0x80000000u : 0u));
    cluster_sync();
    const unsigned v = lane < csize * kWarps ? sm.left[lane] : 0u;
    if (!__any_sync(0xffffffffu, v >> 31)) return true;
    if (warp >= kWarps) return false;
    const int last = (int)__reduce_max_sync(0xffffffffu, v & 0x7fffffffu);
    for (int q = sent; q < last; q++)
        if (lane < csize) announce(at_rank(smem_at(&sm.nearBar[(t0 + q) & 1]), lane), 0u);
    for (int q = due; q < last; q++) {
        // a barrier's last phase is complete only after those before it
        const int par = (int)((t0 + q) & 1);
        if (q + 2 >= last) mbar_wait(smem_at(&sm.nearBar[par]), par ? ph.near1 : ph.near0, kMbarSpins, nullptr);
        if (par) ph.near1 ^= 1u;
        else ph.near0 ^= 1u;
    }
    return false;
}

// The bits of the LGN row of a step into shared memory (thread 0 issues the copy).
__device__ __forceinline__ void fetch_bits(PShared &sm, unsigned *dst, const unsigned *row, int words, int buf) {
    if (threadIdx.x == 0) {
        const unsigned bar = smem_at(&sm.bitBar[buf]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(words * 4) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_at(dst)),
                     "l"(row), "r"(words * 4), "r"(bar)
                     : "memory");
    }
}

// Synapse q's id among a thread's ids in shared memory ([group of four][kCta] from its column).
__device__ __forceinline__ int synapse_id(const int4 *ids, int q) {
    return reinterpret_cast<const int *>(ids + (q >> 2) * kCta)[q & 3];
}

// Which of a neuron's m LGN synapses (in groups of four) received a spike, and the first two words.
__device__ __forceinline__ LgnIn lgn_spikes(const unsigned *bits, const float *__restrict__ lgnSInfo, const int4 *ids,
                                            const float *wts, int m, int groups) {
    LgnIn in{0u, 0.f, 0.f, ids, wts};
    auto bit = [&](int id) { return (bits[id >> 5] >> (id & 31)) & 1u; };
#pragma unroll 2
    for (int g = 0; g < groups; g++) {
        const int4 id = ids[g * kCta];
        in.mask |= (bit(id.x) | bit(id.y) << 1 | bit(id.z) << 2 | bit(id.w) << 3) << (4 * g);
    }
    in.mask &= m < 32 ? (1u << m) - 1u : 0xffffffffu;
    if (in.mask) {
        const unsigned rest = in.mask & (in.mask - 1);
        in.w0 = __ldcg(lgnSInfo + synapse_id(ids, __ffs(in.mask) - 1));
        if (rest) in.w1 = __ldcg(lgnSInfo + synapse_id(ids, __ffs(rest) - 1));
    }
    return in;
}

// Near delivery of step tp from the block's published spikes (near list: the own block alone), four
// conMat rows read together.  Ascending neuron order and the arithmetic of deliver_prev.
template <bool Rng>
__device__ __forceinline__ void deliver_list(const V1Params &P, const TypeConst &tc, long long tp, int b, int local, int i,
                                             bool active, int itype, NState &st, curandStateMRG32k3a &condState, const float4 *unit,
                                             const unsigned *ball) {
    const int lane = threadIdx.x & 31;
    const int bs = P.blockSize, nE = P.nE, ngE = P.ngE, ngI = P.ngI;
    const unsigned wb = ball[lane];
    unsigned nz = __ballot_sync(0xffffffffu, wb != 0);
    float *recNear = nullptr;
    int nDraw = 0, cntE = 0, done = 0;
    if constexpr (Rng) {
        if (P.recNear && active) {
            const long long rs = tp - P.recStep0;
            if (rs >= 0 && rs < P.recSteps) recNear = P.recNear + ((size_t)rs * P.nV1 + i) * P.recCap;
        }
        const unsigned inE = (lane + 1) * 32 <= nE ? 0xffffffffu : (lane * 32 < nE ? (1u << (nE - lane * 32)) - 1u : 0u);
        cntE = __reduce_add_sync(0xffffffffu, __popc(wb & inE));
    }
    if (nz) {
        float lgE[kMaxNG], lhE[kMaxNG], lgI[kMaxNG], lhI[kMaxNG];
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) lgE[ig] = lhE[ig] = lgI[ig] = lhI[ig] = 0.f;
        const float *col = P.conMat + (size_t)b * P.nnbMax * bs * bs + local;
        unsigned cur = 0u;
        int w = 0;
        while (nz | cur) {
            constexpr int kB = 4;
            int j[kB];
            float sv[kB];
#pragma unroll
            for (int k = 0; k < kB; k++) {
                if (!cur && nz) {
                    w = __ffs(nz) - 1;
                    nz &= nz - 1;
                    cur = __shfl_sync(0xffffffffu, wb, w);
                }
                j[k] = cur ? w * 32 + __ffs(cur) - 1 : -1;
                cur &= cur - 1;
                sv[k] = (j[k] >= 0 && active) ? __ldg(col + (size_t)j[k] * bs) : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kB; k++) {
                if (j[k] < 0) break;
                const bool isE = j[k] < nE;
                float strength = sv[k];
                if constexpr (Rng) {
                    if (strength > 0 && P.condRng)
                        strength = near_failure(P, strength, isE, isE ? done : done - cntE, itype, condState, recNear,
                                                nDraw);
                    done++;
                }
                if (strength > 0) {
                    const float4 u = unit[j[k]];
                    const float g[kMaxNG] = {u.x, u.z}, h[kMaxNG] = {u.y, u.w};
#pragma unroll
                    for (int ig = 0; ig < kMaxNG; ig++) {
                        if (isE && ig < ngE) {
                            const float str = strength * tc.pE[ig];
                            lgE[ig] += str * g[ig];
                            lhE[ig] += str * h[ig];
                        }
                        if (!isE && ig < ngI) {
                            const float str = strength * tc.pI[ig];
                            lgI[ig] += str * g[ig];
                            lhI[ig] += str * h[ig];
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int ig = 0; ig < kMaxNG; ig++) {
            st.gE[ig] += lgE[ig]; st.hE[ig] += lhE[ig];
            st.gI[ig] += lgI[ig]; st.hI[ig] += lhI[ig];
        }
    }
    if (Rng && recNear) P.recNearCount[(size_t)(tp - P.recStep0) * P.nV1 + i] = nDraw;
}

// The later (or, sameStep, the same-step) far events of the CTA's spikers of step t (list of its parity),
// by nWarps warps.
__device__ __forceinline__ void push_own(const V1Params &P, long long t, int tSlot, const PShared &sm, int par, int part,
                                         int nWarps, bool sameStep = false) {
    const int n = sm.cnt[par], lane = threadIdx.x & 31;
    for (int c0 = 0; c0 < n; c0 += 32) {
        const int q = c0 + lane;
        const bool in = q < n;
        push_spikers<kPushU>(P, t, tSlot, in ? sm.e0[par][q] : 0,
                             in ? (sameStep ? sm.n1 : sm.deg)[par][q] : 0, in ? sm.si[par][q] : 1.f,
                             in && sm.preE[par][q], sameStep, part, nWarps);
    }
}

// `steps` steps of the patch P from step t0 for CTA `cta` of its nCta CTAs, with the neuron state, the
// generators and (up to mRows) the LGN synapses of its neurons held on the SM.  Threads past
// kCta are push warps.  dyn: LGN weights and ids [mRows][kCta] each (mRows a multiple of 4), then two
// rows of LGN spike bits of bitRoom words (0: the bits are read from global memory).  General:
// patches with more than mRows LGN synapses or with several spikes per step are accepted too.
// Learn: with LGN->V1 plasticity (the weights change in shared memory and go back at the end).  False if a
// barrier gave up.
template <bool Rng, bool General, bool Learn, bool Push>
__device__ __forceinline__ bool persistent_steps(const V1Params &P, long long t0, int steps, int cta, int nCta, int csize,
                                                 const float *__restrict__ lgnRing, const unsigned *__restrict__ lgnBits,
                                                 int lgnSlots, bool deliverFirst, unsigned *barrier, PShared &sm,
                                                 Phases &ph, float *dyn, int mRows, int bitRoom) {
    const int bs = P.blockSize;
    const int nq = (bs + kCta - 1) / kCta;
    const int b = cta / nq, rank = cta % nq;
    const bool pushWarps = Push && blockDim.x > kCta;
    const bool list = P.noDelay && P.nearSelf && csize == nq;
    const bool coupled = P.farOn || (P.noDelay && !list);
    auto cta_sync = [&]() {
        if (pushWarps) asm volatile("bar.sync 0, %0;" ::"n"(2 * kCta) : "memory");
        else neuron_sync();
    };
    // The push warps also push a step's same-step events and arrive at the grid barrier, and the neuron
    // threads do not wait for that: they go on with the next step up to the grid barrier, behind which the push
    // warps have let go of the lists of step s - 1.
    const bool handoff = pushWarps && coupled && list && nCta > 1;
    auto hand_over = [&]() {
        if (handoff) asm volatile("bar.arrive 2, %0;" ::"n"(2 * kCta) : "memory");
        else if (pushWarps && coupled) cta_sync();
    };
    if (pushWarps && threadIdx.x >= kCta) {
        // push warps: one CTA barrier per step hands over the step's spikers
        int slot = far_ring_slot(P, t0);
        const int part = (threadIdx.x - kCta) >> 5;
        cta_sync();
        if (list && csize > 1) cluster_sync();
        for (int s = 0; s < steps && coupled; s++) {
            const int par = (int)((t0 + s) & 1);
            if (handoff) asm volatile("bar.sync 2, %0;" ::"n"(2 * kCta) : "memory");
            else cta_sync();
            if (sm.abortStep == s) break;
            if (handoff) {
                if (sm.cnt[par] > 0) {
                    push_own(P, t0 + s, slot, sm, par, part, kWarps, true);
                    asm volatile("bar.sync 3, %0;" ::"n"(kCta) : "memory");
                }
                if (threadIdx.x == kCta) {
                    sm.cnt[par ^ 1] = 0;
                    if (s + 1 < steps)
                        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(barrier) : "memory");
                }
            }
            push_own(P, t0 + s, slot, sm, par, part, kWarps);
            if (++slot == P.farDepth) slot = 0;
        }
        return leave_block(sm, list, csize, rank, t0, 0, 0, false, ph);
    }
    const int local = rank * kCta + threadIdx.x;
    const bool active = local < bs;
    const int i = b * bs + (active ? local : 0);
    const int itype = type_of(P, active ? local : 0);
    const bool isE = local < P.nE;

    NState st;
    load_state(P, i, st);
    curandStateMRG32k3a condState, noisyState;
    if (Rng && P.condRng && active) condState = P.rGenCond[i];
    if (Rng && P.noiseRng && active) noisyState = P.rNoisy[i];
    const float tonic = active ? P.tonicDep[i] : 0.f;
    const float depC = tonic_current(P, itype, tonic);
    const int m = active ? P.nLGNperV1[i] : 0;
    // this neuron's outgoing far list (static for the run)
    const int farE0 = (P.farOn && active) ? P.farOff[i] : 0;
    const int farDeg = (P.farOn && active) ? P.farOff[i + 1] - farE0 : 0;
    const int farN1 = (P.farOn && active) ? P.farN1[i] : 0;
    const bool isFarPre = P.farOn && active && P.farPre[i];
    // LGN synapses in shared memory, [synapse][kCta] per array from this thread's column
    const bool smemSyn = !General || (P.maxLGN <= mRows && !P.multiSpike);
    const int rows = (P.maxLGN + 3) & ~3;
    float *smW = dyn + threadIdx.x;
    int4 *smI = reinterpret_cast<int4 *>(dyn + (size_t)mRows * kCta) + threadIdx.x;
    unsigned *smB = reinterpret_cast<unsigned *>(dyn + (size_t)2 * mRows * kCta);
    const bool smemBits = P.lgnW <= bitRoom;
    int lgnSlot = (int)(t0 % lgnSlots);
    if (smemSyn) {
        for (int q = 0; q < rows; q++) {
            reinterpret_cast<int *>(smI + (q >> 2) * kCta)[q & 3] = q < m ? __ldg(P.lgnId + (size_t)q * P.nV1 + i) : 0;
            if (q < m) smW[q * kCta] = __ldcg(P.sLGN + (size_t)q * P.nV1 + i);
        }
    }
    // far events of step t0 - 1 that a per-step launch (or the initial spikes) left to push
    if (P.farOn) far_push_list(P, t0 - 1, cta, nCta);
    if (threadIdx.x == 0) {
        sm.cnt[0] = sm.cnt[1] = 0;
        sm.abortStep = -1;
        sm.stop = 0;
    }
    if (threadIdx.x < kMaxType) sm.type[threadIdx.x] = type_const(P, threadIdx.x);
    const TypeConst &tc = sm.type[itype];
    if (list && threadIdx.x < 2 * (kMaxBS / 32)) sm.list.ball[threadIdx.x >> 5][threadIdx.x & 31] = 0u;
    cta_sync();
    if (threadIdx.x == 0 && barrier) {
        __threadfence();
        // the last CTA to come here: everyone has read the list that was left.  A word of its own: step
        // 0 has no wait, so a CTA can arrive at the end of it before another one has come here
        if (atomicAdd(barrier + 1, 1u) + 1u == (unsigned)nCta && P.farOn)
            P.farCount[0] = P.farCount[1] = P.farCount[2] = 0ull;
    }
    if (list) {
        if (csize > 1) cluster_sync();   // the peers run, and are done with an earlier trial's buffers
        if (deliverFirst) {
            const float w = active ? __ldcg(P.sInfo + (size_t)((t0 - 1) & 1) * P.nV1 + i) : 0.f;
            publish_spikes(P, sm, (int)((t0 - 1) & 1), csize, rank, w >= 1.0f, w, isE);
        }
    }
    // ring slots kept incrementally
    int fsT = P.farOn ? far_ring_slot(P, t0) : 0, fsPrev = P.farOn ? far_ring_slot(P, t0 - 1) : 0;
    int t3 = (int)(t0 % 3);
    const bool rec = P.recSpk || P.rec;
    int recSlot = rec ? (int)(t0 % P.recSlots) : 0, recPrev = rec ? (int)((t0 + P.recSlots - 1) % P.recSlots) : 0;
    FFStep ff;
    // waits for other CTAs: the counter of the grid barrier, the limit for spikes
    unsigned *count = barrier && nCta > 1 ? (coupled ? barrier : barrier + 1) : nullptr;
    const int spins = csize > 1 ? (int)min(P.waitSpins / kGridPolls, (long long)kMbarSpins << 8) : kMbarSpins;
    int s = 0;
    int lost = -1;   // 2 x the step whose wait for spikes ran out, + 1 if it was the one for the bits
    float sLast = 0.f;   // the spike word of the step before (Learn)
    // this neuron's learning variables in shared memory behind the spike bits, one column per thread
    LearnVars lv;
    LearnDecay decay;
    if constexpr (Learn) {
        float *col = dyn + (size_t)2 * mRows * kCta + 2 * bitRoom + threadIdx.x;
        lv = LearnVars{col, col + kCta, col + 2 * kCta, col + 3 * kCta, col + 4 * kCta, col + 5 * kCta, smW, kCta};
        decay = learn_decay(P, P.ffT[isE ? 0 : 1]);
        if (active && (isE || P.ffI)) {
            const LearnVars g = learn_vars(P, i, local);
            if (P.ffLearn) {
                *lv.ltd = *g.ltd;
                *lv.trip = *g.trip;
                *lv.total = *g.total;
                *lv.target = *g.target;
            }
            *lv.avg0 = *g.avg0;
            if (isE) *lv.avg1 = *g.avg1;
        }
    }
    if constexpr (Learn) sLast = active && deliverFirst ? __ldcg(P.sInfo + (size_t)((t0 - 1) & 1) * P.nV1 + i) : 0.f;
    if (smemSyn && smemBits) fetch_bits(sm, smB, lgnBits + (size_t)lgnSlot * P.lgnW, P.lgnW, 0);
    for (; s < steps; s++) {
        const long long t = t0 + s;
        const int par = (int)(t & 1);
        const bool dl = s > 0 || deliverFirst;
        const int buf = s & 1;
        if (lost < 0) {
            // step t - 1's spikes and step t's bits: mostly both are there, or come, at the first poll
            const bool spikes = list && dl, copied = smemSyn && smemBits;
            const unsigned nearBar = smem_at(&sm.nearBar[par ^ 1]), bitBar = smem_at(&sm.bitBar[buf]);
            const unsigned nearPar = par ? ph.near0 : ph.near1, bitPar = buf ? ph.bit1 : ph.bit0;
            unsigned ok = 1u;
            if (spikes) ok = mbar_poll(nearBar, nearPar);
            if (copied) ok &= mbar_poll(bitBar, bitPar);
            if (!__all_sync(0xffffffffu, ok)) {
                if (spikes && !mbar_wait(nearBar, nearPar, spins, &sm.stop)) lost = 2 * s;
                else if (copied && !mbar_wait(bitBar, bitPar, kMbarSpins, nullptr)) lost = 2 * s + 1;
                if (lost >= 0) give_up(sm, list ? csize : 1, P.err, count);
            }
            if (spikes && lost != 2 * s) {
                if (par) ph.near0 ^= 1u;
                else ph.near1 ^= 1u;
            }
            if (copied && lost < 0) {
                if (buf) ph.bit1 ^= 1u;
                else ph.bit0 ^= 1u;
            }
        }
        if (!coupled && !list) neuron_sync();
        const int lgnNext = lgnSlot + 1 == lgnSlots ? 0 : lgnSlot + 1;
        const float *lgnSInfo = lgnRing + (size_t)lgnSlot * P.lgnN;
        LgnIn in{};
        if (smemSyn) {
            // the other buffer was read in step s - 1, before the spikes (or barrier) just waited for
            const unsigned *bits = lgnBits + (size_t)lgnSlot * P.lgnW;
            if (smemBits && lost < 0) {
                bits = smB + buf * bitRoom;
                if (s + 1 < steps)
                    fetch_bits(sm, smB + (buf ^ 1) * bitRoom, lgnBits + (size_t)lgnNext * P.lgnW, P.lgnW, buf ^ 1);
            }
            if (active) in = lgn_spikes(bits, lgnSInfo, smI, smW, m, rows >> 2);
        }
        if constexpr (Learn) {   // the filtered rate of learning 1, 2 and 4, advanced over step t - 1
            if (list && dl && P.ffMode != 3 && active && isE) learn_avg_delivery(P, sLast, lv.avg0, lv.avg1, lv.avg0);
        }
        if (list && dl)
            deliver_list<Rng>(P, tc, t - 1, b, local, i, active, itype, st, condState, sm.list.unit[par ^ 1],
                              sm.list.ball[par ^ 1]);
        auto feed_forward = [&]() {
            if (!active || (General && P.multiSpike)) return;
            if (smemSyn)
                step_feedforward<Rng, true>(P, tc, t, i, itype, tonic, depC, m, lgnSInfo, st, condState, noisyState, ff, in);
            else
                step_feedforward<Rng, false>(P, tc, t, i, itype, tonic, depC, m, lgnSInfo, st, condState, noisyState, ff);
        };
        // failure draws of the near synapses precede those of the LGN synapses: with a general
        // neighbour list they come after the barrier
        const bool ffEarly = list || !dl;
        if (ffEarly) feed_forward();
        if (s > 0 && (coupled || (s == 1 && count))) {
            // behind every CTA's arrival of step s - 1; uncoupled, behind the start of every CTA
            if (!meet(count, (unsigned)nCta * (coupled ? (unsigned)s : 1u), lost >= 0, P.err, P.waitSpins)) {
                if (lost < 0) give_up(sm, list ? csize : 1, P.err, count);
                if (threadIdx.x == 0) sm.abortStep = s;
                hand_over();
                break;
            }
        } else if (lost >= 0 && list && !coupled && (s > 0 || !count)) {
            break;
        }
        if (dl) {
            if (!list) {
                deliver_prev<Rng>(P, t - 1, b, local, i, active, itype, st, condState, sm.near, P.farOn ? fsPrev : -1);
            } else if (active) {
                if (P.farClass) {
                    FarIn fin;
                    far_fetch(P, fsPrev, t3 == 0 ? 2 : t3 - 1, i, fin);
                    far_apply(P, fsPrev, i, fin, st);
                }
                if (P.rec) record_conductances(P, recPrev, i, st);
            }
        }
        if (!ffEarly) feed_forward();
        float sInfo = 0.f;
        const float vBefore = st.v;
        if (active && !(General && P.multiSpike)) sInfo = step_membrane(P, tc, depC, ff, st);
        if (General && active && P.multiSpike)
            sInfo = step_multi<Rng>(P, t, i, itype, tonic, depC, m, lgnSInfo, st, condState, noisyState);
        const bool spk = active && sInfo >= 1.0f;
        if (list && s + 1 < steps) publish_spikes(P, sm, par, csize, rank, spk, sInfo, isE);
        if constexpr (Learn) {
            sLast = sInfo;
            if (active && P.ffLearn)
                learn_ff(P, i, local, m, sInfo, lgnSInfo, P.ffPreRing + (size_t)lgnSlot * P.ffTypes * 2 * P.lgnN, P.lgnN, lv,
                         decay, &in);
        }
        // a neuron that enters the last tenth below its threshold will likely spike some steps from now:
        // what its delivery and its same-step push wait for is then already in L2
        if (active && !spk) {
            const float near = tc.level.y - 0.1f * (tc.level.y - tc.level.x);
            if (vBefore < near && st.v >= near) prefetch_spiker(P, b, local, farE0, farN1);
        }
        if (spk && farDeg > farN1) prefetch_far(P, farE0 + farN1, farDeg - farN1);
        if (P.farOn) {
            if (spk && farDeg > 0) {
                const int q = atomicAdd(&sm.cnt[par], 1);
                sm.e0[par][q] = farE0;
                sm.deg[par][q] = farDeg;
                sm.n1[par][q] = farN1;
                sm.si[par][q] = sInfo;
                sm.preE[par][q] = isE;
            }
            far_same_step(P, t, t3, fsT, spk, sInfo, isFarPre, isE, farE0, handoff ? 0 : farN1,
                          cta == 0 && threadIdx.x == 0);
        }
        // spike words other CTAs read in the next step (general neighbour lists) come before the arrival
        const bool storeFirst = !list || (General && P.multiSpike);
        if (storeFirst && active && !(General && P.multiSpike)) store_step(P, t, i, sInfo, ff.depOut, st, recSlot);
        if (handoff) {
            hand_over();
        } else if (coupled) {
            cta_sync();
            if (threadIdx.x == 0) {
                sm.cnt[par ^ 1] = 0;   // pushed: step t + 1's spikers go there
                if (s + 1 < steps)
                    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(barrier) : "memory");
            }
        }
        if (!storeFirst && active) store_step(P, t, i, sInfo, ff.depOut, st, recSlot);
        if (P.spikeCount && spk) atomicAdd(P.spikeCount + i, (unsigned)floorf(sInfo));
        if (P.farOn && !pushWarps) push_own(P, t, fsT, sm, par, threadIdx.x >> 5, kWarps);
        lgnSlot = lgnNext;
        recPrev = recSlot;
        if (++recSlot == P.recSlots) recSlot = 0;
        fsPrev = fsT;
        if (++fsT == P.farDepth) fsT = 0;
        t3 = t3 == 2 ? 0 : t3 + 1;
    }
    if constexpr (Learn) {
        if (active && P.ffLearn)
            for (int q = 0; q < m; q++) P.sLGNw[(size_t)q * P.nV1 + i] = smW[q * kCta];
        if (active && (isE || P.ffI)) {
            const LearnVars g = learn_vars(P, i, local);
            if (P.ffLearn) {
                *g.ltd = *lv.ltd;
                *g.trip = *lv.trip;
                *g.total = *lv.total;
            }
            *g.avg0 = *lv.avg0;
            if (isE) *g.avg1 = *lv.avg1;
        }
    }
    if (active) {
        store_state(P, i, st);
        if (!(General && P.multiSpike)) P.dep[i] = ff.depOut;
        if (Rng && P.condRng) P.rGenCond[i] = condState;
        if (Rng && P.noiseRng) P.rNoisy[i] = noisyState;
    }
    const int sent = min(s, steps - 1);
    if (smemSyn && smemBits && threadIdx.x < 32 && (s < steps || lost >= 0)) {
        // gave up: no CTA ends under a copy into it.  Copies are asked for a step ahead, and not any more once lost
        const int q = lost < 0 ? s + 1 : lost >> 1;
        if (q < steps) mbar_wait(smem_at(&sm.bitBar[q & 1]), q & 1 ? ph.bit1 : ph.bit0, kMbarSpins, nullptr);
    }
    return leave_block(sm, list, csize, rank, t0, sent, lost < 0 ? sent : (lost - 1) >> 1, s < steps || lost >= 0, ph);
}

// CTAs per cluster, as launched: a tool that relaunches the kernel without clusters gets the
// general path.
__device__ __forceinline__ int cluster_ctas() {
    int n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n;
}

// K steps of one patch in one cooperative launch.
template <bool Rng, bool Learn>
__global__ void __launch_bounds__(2 * kCta, 1) v1_persistent_kernel(V1Params P, const long long *stepBase, int K,
                                                                    const float *__restrict__ lgnRing,
                                                                    const unsigned *__restrict__ lgnBits, int lgnSlots,
                                                                    int deliverFirst, unsigned *barrier, int bitRoom) {
    __shared__ PShared sm;
    extern __shared__ __align__(16) float lgnSm[];
    Phases ph;
    const int csize = cluster_ctas();
    init_barriers(sm, csize);
    persistent_steps<Rng, false, Learn, true>(P, *stepBase, K, blockIdx.x, gridDim.x, csize, lgnRing, lgnBits, lgnSlots,
                                 deliverFirst != 0, barrier, sm, ph, lgnSm, (P.maxLGN + 3) & ~3, bitRoom);
}

// rand_spInit (src/coredynamics.cu:5-146) for a network without initial spikes: seeds the
// two per-neuron generators and consumes the uniforms the reference draws while it fills
// the spike history (one, then one per older slot).
__global__ void v1_rng_init_kernel(curandStateMRG32k3a *cond, curandStateMRG32k3a *noisy,
                                   unsigned long long seed, int nV1, int trainDepth) {
    int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nV1) return;
    curandStateMRG32k3a a, b;
    mrg_seed(seed, id, &a);
    mrg_seed(seed, (unsigned long long)nV1 + id, &b);
    (void)curand_uniform(&a);
    for (int q = trainDepth - 1; q > 0; q--) (void)curand_uniform(&a);
    cond[id] = a;
    noisy[id] = b;
}

// ---- initial spikes (spE0/spI0 > 0) ----
// rand_spInit (src/coredynamics.cu:5-146) with initial spikes, one CTA per block of neurons:
// neuron id spikes with chance sp0[type][nLGN > SCsplit ? 0 : 1] at a uniform time tsp of the
// step before the first (v = vR, tBack and the AdEx w advanced over the rest of that step),
// then the history slots depth-1 .. 1 of the spike-word ring are filled with spikes of the
// same chance outside the refractory period.  H [depth][nV1] receives the spike words (slot 0:
// the initial ones).  ogTab/ohTab [nblock][nE*ngE + nI*ngI] receive output_g/h of the initial
// spikers as the reference writes them for the step's compacted spiker list (E then I, each
// numbered within its block); the reference numbers them in the order its atomicAdd_block
// calls return, which the hardware does not fix, and this kernel numbers them by thread index.
__global__ void __launch_bounds__(1024) v1_sp_init_kernel(V1Params P, unsigned long long seed, int depth, Sp0 sp0,
                                                          int SCsplit, float *H, float *ogTab, float *ohTab,
                                                          float *recU, unsigned *recNU) {
    __shared__ int sCnt[2][32];
    const int bs = P.blockSize, nV1 = P.nV1;
    const int b = blockIdx.x, local = threadIdx.x;
    const bool active = local < bs;
    const int id = b * bs + (active ? local : 0);
    const int itype = type_of(P, active ? local : 0);
    const float dt = P.dt;
    float sInfo = -1.f;
    if (active) {
        curandStateMRG32k3a a, nz;
        mrg_seed(seed, id, &a);
        mrg_seed(seed, (unsigned long long)nV1 + id, &nz);
        float *ru = recU ? recU + (size_t)id * 2 * depth : nullptr;
        int nu = 0;
        auto draw = [&]() {
            const float u = curand_uniform(&a);
            if (ru) ru[nu] = u;
            nu++;
            return u;
        };
        const float r0 = draw();
        const float chance = sp0.c[itype * 2 + (P.nLGNperV1[id] > SCsplit ? 0 : 1)];
        const float tRef = P.tRef[itype];
        float v = P.v[id];
        float ref = 0.f;
        sInfo = v;
        if (chance > 0 && r0 < chance) {
            const float tsp = draw();
            sInfo = 1.0f + tsp;
            const float tb = tRef - (1 - tsp) * dt;
            if (tb > 0) P.tBack[id] = tb;
            const float v0 = P.vR[itype];
            v = v0;
            P.v[id] = v0;
            if (P.iModel == 1) {
                const float tw = P.tau_w[itype];
                const float A = P.a[itype] * (v0 - P.vL) * tw;
                const float w0 = P.w[id] + P.b[itype];
                P.w[id] = (w0 - A) * expf(-dt * (1 - tsp) / tw) + A;
            }
            ref = (1 - tsp) * dt + tRef - dt;
        }
        H[id] = sInfo;
        for (int q = depth - 1; q > 0; q--) {
            float word;
            if (ref < dt) {
                if (ref < 0) ref = 0;
                if (draw() < chance * (dt - ref) / dt) {
                    const float tsp = draw() * (dt - ref) / dt;
                    word = 1.0f + tsp;
                    ref = tRef + (1 - tsp) * dt;
                } else {
                    word = v;
                }
            } else {
                word = P.vR[itype];
            }
            H[(size_t)q * nV1 + id] = word;
            ref -= dt;
        }
        P.rGenCond[id] = a;
        P.rNoisy[id] = nz;
        if (recNU) recNU[id] = (unsigned)nu;
    }
    if (!ogTab) return;
    // block-wide numbering of the initial E and I spikers in thread order
    const bool isE = local < P.nE;
    const bool spk = active && sInfo >= 1.0f;
    const int lane = local & 31, warp = local >> 5, nw = (blockDim.x + 31) >> 5;
    const unsigned bE = __ballot_sync(0xffffffffu, spk && isE);
    const unsigned bI = __ballot_sync(0xffffffffu, spk && !isE);
    if (lane == 0) {
        sCnt[0][warp] = __popc(bE);
        sCnt[1][warp] = __popc(bI);
    }
    __syncthreads();
    int before = 0, nE = 0, nI = 0;
    for (int w2 = 0; w2 < nw; w2++) {
        if (w2 < warp) before += isE ? sCnt[0][w2] : sCnt[1][w2];
        nE += sCnt[0][w2];
        nI += sCnt[1][w2];
    }
    if (!spk) return;
    const int sid = before + __popc((isE ? bE : bI) & ((1u << lane) - 1u));
    const size_t base = (size_t)b * (P.nE * P.ngE + P.nI * P.ngI);
    const float tsp = (sInfo - 1) * dt;
    const int ng = isE ? P.ngE : P.ngI;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ng) {
            float g = 0.f, h = 0.f;
            if (isE) cond_input(P.condE, g, h, 1.f, dt - tsp, ig);
            else cond_input(P.condI, g, h, 1.f, dt - tsp, ig);
            const size_t r = isE ? (size_t)ig * nE + sid : (size_t)ig * nI + (size_t)nE * P.ngE + sid;
            ogTab[base + r] = g;
            ohTab[base + r] = h;
        }
    }
}

// The near delivery that runs once before the first step when there are initial spikes
// (noDelay = 1): recal_G_mat_nd (src/coredynamics.cu:2366-2608) as src/patch.cu:5750-5758
// launches it, on the history slot depth-1 of the spike-word ring, reading output_g/h at
// the per-neuron offsets (block, E: i*ngE, I: nE*ngE + (i-nE)*ngI) of the table that
// v1_sp_init_kernel wrote in the compacted layout; the sums are added to gE/hE/gI/hI.
__global__ void __launch_bounds__(1024) v1_sp_near_kernel(V1Params P, const float *Hlast, const float *ogTab,
                                                          const float *ohTab, float *recZ, unsigned *recNZ,
                                                          int cap) {
    const int bs = P.blockSize, nV1 = P.nV1;
    const int b = blockIdx.x, local = threadIdx.x;
    if (local >= bs) return;
    const int ipost = b * bs + local;
    const int itype = type_of(P, local);
    const int ngE = P.ngE, ngI = P.ngI;
    const int ncb = P.nE * ngE + P.nI * ngI;
    float lgE[kMaxNG], lhE[kMaxNG], lgI[kMaxNG], lhI[kMaxNG], ipE[kMaxNG], ipI[kMaxNG];
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        lgE[ig] = lhE[ig] = lgI[ig] = lhI[ig] = 0.f;
        ipE[ig] = ig < ngE ? P.pE[itype * ngE + ig] : 0.f;
        ipI[ig] = ig < ngI ? P.pI[itype * ngI + ig] : 0.f;
    }
    curandStateMRG32k3a cs = P.rGenCond[ipost];
    int nz = 0;
    for (int ib = 0; ib < P.nNearNB[b]; ib++) {
        const int bid = P.nbId[b * P.nnbMax + ib];
        const float *col = P.conMat + ((size_t)(b * P.nnbMax + ib) * bs) * bs + local;
        for (int i = 0; i < bs; i++) {
            float strength = col[(size_t)i * bs];
            if (!(strength != 0 && Hlast[(size_t)bid * bs + i] > 0)) continue;
            const int jtype = type_of(P, i);
            const float p = P.synFail[jtype * P.nType + itype];
            if (p > 0) {
                const float normed_std = sqrtf(p * (1 - p) / P.synPerCon[jtype * P.nType + itype]);
                const float rnd = curand_normal(&cs);
                if (recZ) {
                    if (nz < cap) recZ[(size_t)ipost * cap + nz] = rnd;
                    else atomicOr(P.err, kErrRecordOverflow);
                }
                nz++;
                strength *= 1 - p + normed_std * rnd;
            }
            if (strength > 0) {
                const bool isE = i < P.nE;
                const size_t base = (size_t)bid * ncb + (isE ? (size_t)i * ngE : (size_t)P.nE * ngE + (size_t)(i - P.nE) * ngI);
#pragma unroll
                for (int ig = 0; ig < kMaxNG; ig++) {
                    if (isE && ig < ngE) {
                        const float str = strength * ipE[ig];
                        lgE[ig] += str * ogTab[base + ig];
                        lhE[ig] += str * ohTab[base + ig];
                    }
                    if (!isE && ig < ngI) {
                        const float str = strength * ipI[ig];
                        lgI[ig] += str * ogTab[base + ig];
                        lhI[ig] += str * ohTab[base + ig];
                    }
                }
            }
        }
    }
    P.rGenCond[ipost] = cs;
    if (recNZ) recNZ[ipost] = (unsigned)nz;
#pragma unroll
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig < ngE) { P.gE[(size_t)ig * nV1 + ipost] += lgE[ig]; P.hE[(size_t)ig * nV1 + ipost] += lhE[ig]; }
        if (ig < ngI) { P.gI[(size_t)ig * nV1 + ipost] += lgI[ig]; P.hI[(size_t)ig * nV1 + ipost] += lhI[ig]; }
    }
}

// Delayed events of the history, one thread per presynaptic neuron.  Far synapses
// (fill_fSpikeTrain before the loop, src/patch.cu:5806-5846) see the history slot depth-1 as
// step -1: its events arriving in step -1 go to ring slot farDepth-1 (delivered before the
// first step), and the neuron joins step -1's far spiker list, from which step 0 pushes the
// later arrivals.  Delayed near synapses (noDelay = 0) follow recal_G_mat's reads of the
// ring: before the loop (current slot 0, src/patch.cu:5760-5770) slot 0 is step -1 and slot
// s >= 1 step s-depth-1, and only arrivals in step -1 count; in the loop slot s is step
// s-depth until it is overwritten, so slots 1 .. depth-2 push their arrivals in steps >= 0
// here (slot depth-1's come from step -1's list as above).
__global__ void v1_sp_push_kernel(V1Params P, const float *H, int depth) {
    const int nV1 = P.nV1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nV1) return;
    const float sLast = H[(size_t)(depth - 1) * nV1 + i];
    const int e0 = P.farOff[i], deg = P.farOff[i + 1] - e0;
    if (sLast > 1.0f && P.farPre[i]) P.farFlag[2] = 1;
    if (sLast >= 1.0f && deg > 0) {
        const int pos = (int)(atomicAdd(P.farCount + 2, (1ull << 32) | (unsigned)deg) >> 32);
        P.farList[(size_t)2 * nV1 + pos] = make_int4(i, e0, deg, __float_as_int(sLast));
    }
    for (int e = e0; e < e0 + deg; e++) {
        const int post = P.farPost[e];
        const float f = P.farStr[e];
        const int sp = P.farSteps[e];
        const float frac = P.farFrac[e];
        const int steps = sp & 0xffff;
        if (!((sp >> 24) & 1)) {
            if (sLast >= 1.0f && steps <= 1) far_event(P, -1, far_ring_slot(P, -1), i, sLast, post, f, sp, frac, steps);
            continue;
        }
        for (int q = 0; q < depth; q++) {
            const float w = H[(size_t)q * nV1 + i];
            if (w < 1.0f) continue;
            const long long th = q == 0 ? -1 : (long long)q - depth - 1;
            const long long k = th + steps + 1;
            if (k == 0 || k == 1) far_event(P, th, far_ring_slot(P, th), i, w, post, f, sp, frac, (int)k);
        }
        for (int q = 1; q < depth - 1; q++) {
            const float w = H[(size_t)q * nV1 + i];
            if (w < 1.0f) continue;
            const long long th = (long long)q - depth;
            for (int k = 0; k < 2; k++)
                if (k <= steps && th + steps - k >= 0) far_event(P, th, far_ring_slot(P, th), i, w, post, f, sp, frac, k);
        }
    }
}

// Adds ring slot farDepth-1 (arrivals in step -1) to the conductances and clears it: delayed
// near events as recal_G_mat adds them, then the far events as sum_G does when some far
// presynaptic neuron spiked in step -1 (src/patch.cu:5806-5846).
__global__ void v1_sp_consume_kernel(V1Params P) {
    const int nV1 = P.nV1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nV1) return;
    const int ngE = P.ngE, ns = P.ngE + P.ngI;
    const size_t slot = (size_t)(P.farDepth - 1) * ns * 2 * nV1;
    for (int pass = 0; pass < 2; pass++) {
        unsigned long long *acc = pass == 0 ? (P.nearOn ? P.nearAcc : nullptr) : (P.farClass ? P.farAcc : nullptr);
        if (!acc) continue;
        const bool add = pass == 0 || P.farFlag[2] != 0;
        acc += slot;
        for (int q = 0; q < ns; q++) {
            unsigned long long *pg = acc + (size_t)(2 * q) * nV1 + i;
            unsigned long long *ph = acc + (size_t)(2 * q + 1) * nV1 + i;
            const unsigned long long ug = *pg, uh = *ph;
            *pg = 0ull;
            *ph = 0ull;
            if (!add) continue;
            const float fg = far_from_fixed(ug), fh = far_from_fixed(uh);
            if (q < ngE) {
                P.gE[(size_t)q * nV1 + i] += fg;
                P.hE[(size_t)q * nV1 + i] += fh;
            } else {
                P.gI[(size_t)(q - ngE) * nV1 + i] += fg;
                P.hI[(size_t)(q - ngE) * nV1 + i] += fh;
            }
        }
    }
}

__global__ void advance_step_kernel(long long *stepBase, int k) { *stepBase += k; }

// Full-step decay factors, evaluated with the same expressions as cond_decay (one thread).
__global__ void step_decay_kernel(Cond cFF, Cond cE, Cond cI, float dt, StepDecay *out) {
    if (threadIdx.x != 0) return;
    const Cond *cs[3] = {&cFF, &cE, &cI};
    for (int k = 0; k < 3; k++) {
        for (int ig = 0; ig < kMaxNG; ig++) {
            out[k].etr[ig] = expf(-dt / cs[k]->rise[ig]);
            out[k].etd[ig] = expf(-dt / cs[k]->decay[ig]);
        }
    }
}

// Compares div_known with the division for every significand x in [1, 2) and every time of the
// kernel conds[blockIdx.y]; a difference clears its flag.
__global__ void __launch_bounds__(256) quick_division_kernel(Cond c0, Cond c1, Cond c2, int n0, int n1, int n2, int *ok) {
    const Cond &c = blockIdx.y == 0 ? c0 : (blockIdx.y == 1 ? c1 : c2);
    const int n = blockIdx.y == 0 ? n0 : (blockIdx.y == 1 ? n1 : n2);
    const float x = __uint_as_float(0x3f800000u + blockIdx.x * blockDim.x + threadIdx.x);
    bool same = true;
    for (int ig = 0; ig < kMaxNG; ig++) {
        if (ig >= n) break;
        same = same && div_known(x, c.rise[ig], c.riseHi[ig], c.riseLo[ig], 1) == x / c.rise[ig];
        same = same && div_known(x, c.decay[ig], c.decayHi[ig], c.decayLo[ig], 1) == x / c.decay[ig];
    }
    if (!same) ok[blockIdx.y] = 0;
}

cudaError_t compute_step_decay(V1Params &p, cudaStream_t st) {
    struct Out {
        StepDecay dec[3];
        int ok[3];
    } h, *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(Out));
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(d, 1, sizeof(Out), st);
    step_decay_kernel<<<1, 32, 0, st>>>(p.condFF, p.condE, p.condI, p.dt, d->dec);
    if (e == cudaSuccess) e = cudaGetLastError();
    quick_division_kernel<<<dim3((1 << 23) / 256, 3), 256, 0, st>>>(p.condFF, p.condE, p.condI, p.ngFF, p.ngE, p.ngI,
                                                                  d->ok);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) return e;
    p.decFF = h.dec[0];
    p.decE = h.dec[1];
    p.decI = h.dec[2];
    // times far from 1 could take the products of the check out of the normal range
    auto plain = [](const Cond &c, int n) {
        bool in = true;
        for (int k = 0; k < n; k++) in = in && c.rise[k] > 1e-6f && c.rise[k] < 1e6f && c.decay[k] > 1e-6f && c.decay[k] < 1e6f;
        return in;
    };
    p.condFF.quick = h.ok[0] != 0 && plain(p.condFF, p.ngFF);
    p.condE.quick = h.ok[1] != 0 && plain(p.condE, p.ngE);
    p.condI.quick = h.ok[2] != 0 && plain(p.condI, p.ngI);
    return cudaSuccess;
}

// The random-number paths are needed when a draw can change a result (the draws are then
// also recorded when recording is on).
static bool needs_rng(const V1Params &p) { return p.condRng || p.noiseRng; }

cudaError_t launch_v1_step(const V1Params &p, const long long *stepBase, int stepOffset,
                           const float *lgnSInfo, int lgnSlots, int deliverPrev, int doStep,
                           cudaStream_t st) {
    const int nq = (p.blockSize + kCta - 1) / kCta;
    if (needs_rng(p))
        v1_step_kernel<true><<<p.nblock * nq, kCta, 0, st>>>(p, stepBase, stepOffset, lgnSInfo, lgnSlots,
                                                             deliverPrev, doStep);
    else
        v1_step_kernel<false><<<p.nblock * nq, kCta, 0, st>>>(p, stepBase, stepOffset, lgnSInfo, lgnSlots,
                                                              deliverPrev, doStep);
    return cudaGetLastError();
}

// A launch of `grid` CTAs in clusters of csize, cooperative or not.
struct CoopLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    CoopLaunch(int grid, int threads, size_t smem, int csize, cudaStream_t st, bool coop = true) {
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = csize;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.attrs = coop ? attr : attr + 1;
        cfg.numAttrs = (coop ? 1 : 0) + (csize > 1 ? 1 : 0);
    }
};

// CTAs of a kernel that can be resident at once, in whole clusters.
template <class Kern>
static int resident_ctas(Kern kern, int threads, size_t smem, int csize, int device) {
    int n = 0;
    if (csize > 1) {
        CoopLaunch cl(csize, threads, smem, csize, nullptr, false);
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cl.cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n * csize;
    }
    int sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n * sms;
}

// Dynamic shared memory of the persistent kernel: weights and ids of the LGN synapses of each thread,
// two rows of LGN spike bits.
static int v1_persistent_bits(const V1Params &p) { return p.lgnW <= kMaxBitWords ? p.lgnW : 0; }
static size_t v1_persistent_smem(const V1Params &p) {
    return ((size_t)2 * ((p.maxLGN + 3) & ~3) * kCta + 2 * v1_persistent_bits(p) + (p.ffMode ? kLearnVars * kCta : 0)) *
           sizeof(float);
}

using PersistentKernel = void (*)(V1Params, const long long *, int, const float *, const unsigned *, int, int, unsigned *, int);
static PersistentKernel persistent_kernel(const V1Params &p) {
    if (p.ffMode) return needs_rng(p) ? v1_persistent_kernel<true, true> : v1_persistent_kernel<false, true>;
    return needs_rng(p) ? v1_persistent_kernel<true, false> : v1_persistent_kernel<false, false>;
}

// The shape of the persistent launch: a block's CTAs as a cluster, with push warps when there are
// far synapses and every CTA still finds an SM; else without push warps (two CTAs share an SM);
// else single CTAs, whose near delivery then goes through global memory.
bool v1_persistent_shape(const V1Params &p, int device, int *cluster, int *threads) {
    const int nq = (p.blockSize + kCta - 1) / kCta;
    const int n = p.nblock * nq;
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
    if (!coop || p.maxLGN > kMaxLgnReg) return false;
    const int maxDyn = (int)(((size_t)2 * kMaxLgnReg * kCta + 2 * kMaxBitWords + kLearnVars * kCta) * sizeof(float));
    const PersistentKernel kern = persistent_kernel(p);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, maxDyn) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const size_t dyn = v1_persistent_smem(p);
    const int shapes[3][2] = {{nq, 2 * kCta}, {nq, kCta}, {1, kCta}};
    for (int k = p.farOn ? 0 : 1; k < 3; k++) {
        if (resident_ctas(kern, shapes[k][1], dyn, shapes[k][0], device) < n) continue;
        *cluster = shapes[k][0];
        *threads = shapes[k][1];
        return true;
    }
    return false;
}

cudaError_t launch_v1_persistent(const V1Params &p, const long long *stepBase, int K, const float *lgnRing,
                                 const unsigned *lgnBits, int lgnSlots, int deliverFirst, unsigned *barrier,
                                 cudaStream_t st) {
    const int nq = (p.blockSize + kCta - 1) / kCta;
    CoopLaunch cl(p.nblock * nq, p.threads, v1_persistent_smem(p), p.cluster, st, barrier != nullptr);
    if (barrier) {
        const cudaError_t e = cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), st);
        if (e != cudaSuccess) return e;
    }
    return cudaLaunchKernelEx(&cl.cfg, persistent_kernel(p), p, stepBase, K, lgnRing, lgnBits, lgnSlots, deliverFirst,
                              barrier, v1_persistent_bits(p));
}

cudaError_t launch_v1_rng_init(curandStateMRG32k3a *cond, curandStateMRG32k3a *noisy,
                               unsigned long long seed, int nV1, int trainDepth, cudaStream_t st) {
    v1_rng_init_kernel<<<(nV1 + 127) / 128, 128, 0, st>>>(cond, noisy, seed, nV1, trainDepth);
    return cudaGetLastError();
}

cudaError_t launch_v1_sp_init(const V1Params &p, unsigned long long seed, int depth, const Sp0 &sp0, int SCsplit,
                              float *H, float *ogTab, float *ohTab, float *recU, unsigned *recNU, cudaStream_t st) {
    const int threads = (p.blockSize + 31) / 32 * 32;
    v1_sp_init_kernel<<<p.nblock, threads, 0, st>>>(p, seed, depth, sp0, SCsplit, H, ogTab, ohTab, recU, recNU);
    return cudaGetLastError();
}

cudaError_t launch_v1_sp_near(const V1Params &p, const float *Hlast, const float *ogTab, const float *ohTab,
                              float *recZ, unsigned *recNZ, int cap, cudaStream_t st) {
    const int threads = (p.blockSize + 31) / 32 * 32;
    v1_sp_near_kernel<<<p.nblock, threads, 0, st>>>(p, Hlast, ogTab, ohTab, recZ, recNZ, cap);
    return cudaGetLastError();
}

cudaError_t launch_v1_sp_events(const V1Params &p, const float *H, int depth, cudaStream_t st) {
    const int n = (p.nV1 + 255) / 256;
    v1_sp_push_kernel<<<n, 256, 0, st>>>(p, H, depth);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    v1_sp_consume_kernel<<<n, 256, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_advance_step(long long *stepBase, int k, cudaStream_t st) {
    advance_step_kernel<<<1, 1, 0, st>>>(stepBase, k);
    return cudaGetLastError();
}

// ---- batched trials ----
// One step of every active (trial, CTA) tile of a batch.  Each CTA copies its trial's
// parameter block to shared memory and runs the same step body as the per-step kernel with
// the trial's own CTA index and count, so each trial computes exactly what it would alone.
// Finished trials have no tiles in the list (the host rebuilds it between chunks); a tile
// whose trial ends inside the chunk returns at its last step.
template <bool Rng, int MinB>
__global__ void __launch_bounds__(kCta, MinB) v1_batch_step_kernel(const BatchTrial *__restrict__ trials,
                                                                   const int2 *__restrict__ tiles,
                                                                   const int *__restrict__ nTiles,
                                                                   int stepOffset) {
    __shared__ Smem sm;
    __shared__ __align__(16) BatchTrial sT;
    if ((int)blockIdx.x >= *nTiles) return;
    const int2 tile = tiles[blockIdx.x];
    const int *src = reinterpret_cast<const int *>(trials + tile.x);
    int *dst = reinterpret_cast<int *>(&sT);
    for (int w = threadIdx.x; w < (int)(sizeof(BatchTrial) / sizeof(int)); w += kCta) dst[w] = src[w];
    __syncthreads();
    const long long t = *sT.step + stepOffset;
    if (t >= sT.tEnd) return;
    v1_step_body<Rng>(sT.v, t, tile.y, sT.nCta, sT.lgnRing, sT.lgnSlots, t >= sT.tDeliverFrom ? 1 : 0, 1, sm);
}

// Batched trials in one cooperative launch per chunk: the grid is split into slots of
// slotCtas CTAs (the largest trial's CTA count); slot s runs active trials s, s + nSlots, ...
// one after the other, each for its steps of the chunk, with the trial's state in registers
// and a barrier among the trial's own CTAs between steps (no grid-wide barrier: trials are
// independent).  The step is the single patch's (persistent_steps), so every trial computes
// what the per-step batch and pv1_run compute for it.  Push: with push warps, one CTA per SM (batches whose
// trials all have far synapses; the host chooses the form).
template <bool Rng, bool General, bool Push>
__global__ void __launch_bounds__(Push ? 2 * kCta : kCta, Push ? 1 : 2)
    v1_batch_persistent_kernel(const BatchTrial *__restrict__ trials, const int *__restrict__ activeList,
                               const int *__restrict__ nActive, int slotCtas, int nSlots, int K, unsigned *barriers) {
    __shared__ PShared sm;
    __shared__ __align__(16) BatchTrial sT;
    extern __shared__ __align__(16) float dyn[];   // LGN synapses: weights, ids [kBatchLgn][kCta] each; spike bits
    Phases ph;
    const int csize = cluster_ctas();
    init_barriers(sm, csize);
    const int slot = blockIdx.x / slotCtas, c = blockIdx.x % slotCtas;
    const int na = *nActive;
    for (int j = slot; j < na; j += nSlots) {
        const int q = activeList[j];
        if (q < 0) continue;  // a slot's schedule ended (one-launch sweep)
        __syncthreads();
        const int *src = reinterpret_cast<const int *>(trials + q);
        int *dst = reinterpret_cast<int *>(&sT);
        for (int w = threadIdx.x; w < (int)(sizeof(BatchTrial) / sizeof(int)); w += blockDim.x) dst[w] = src[w];
        __syncthreads();
        if (c >= sT.nCta) continue;
        const long long t0 = *sT.step;
        const long long left = sT.tEnd - t0;
        const int steps = left < K ? (int)left : K;
        if (steps <= 0) continue;
        // a trial whose barrier gave up ends the slot: its cluster's CTAs leave it a step apart
        if (!persistent_steps<Rng, General, false, Push>(sT.v, t0, steps, c, sT.nCta, csize, sT.lgnRing, sT.lgnBits, sT.lgnSlots,
                                            t0 >= sT.tDeliverFrom, barriers + 2 * q, sm, ph, dyn, kBatchLgn, kBatchBits))
            return;
    }
}


using BatchKernel = void (*)(const BatchTrial *, const int *, const int *, int, int, int, unsigned *);
template <bool Push>
static BatchKernel batch_kernel_of(bool rng, bool general) {
    if (general) return rng ? v1_batch_persistent_kernel<true, true, Push> : v1_batch_persistent_kernel<false, true, Push>;
    return rng ? v1_batch_persistent_kernel<true, false, Push> : v1_batch_persistent_kernel<false, false, Push>;
}
static BatchKernel batch_kernel(bool rng, bool general, bool push) {
    return push ? batch_kernel_of<true>(rng, general) : batch_kernel_of<false>(rng, general);
}

// Whether a trial needs the general kernel: LGN lists past kBatchLgn or several spikes per step.
bool v1_batch_general(const V1Params &p) { return p.multiSpike || p.maxLGN > kBatchLgn; }

int v1_batch_persistent_capacity(bool rng, bool general, bool push, int device, int csize) {
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) return 0;
    BatchKernel k = batch_kernel(rng, general, push);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchDyn) != cudaSuccess) return 0;
    return resident_ctas(k, push ? 2 * kCta : kCta, kBatchDyn, csize, device);
}

cudaError_t launch_v1_batch_persistent(const BatchTrial *trials, const int *activeList, const int *nActive,
                                       int slotCtas, int nSlots, int K, unsigned *barriers, int nTrials, bool rng,
                                       bool general, bool push, int csize, cudaStream_t st) {
    if (nSlots <= 0 || slotCtas <= 0 || csize <= 0 || slotCtas % csize) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(barriers, 0, (size_t)2 * nTrials * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    CoopLaunch cl(nSlots * slotCtas, push ? 2 * kCta : kCta, kBatchDyn, csize, st);
    return cudaLaunchKernelEx(&cl.cfg, batch_kernel(rng, general, push), trials, activeList, nActive, slotCtas, nSlots, K,
                              barriers);
}

template <bool Rng>
static cudaError_t launch_batch_variant(int minB, const BatchTrial *trials, const int2 *tiles,
                                        const int *nTiles, int grid, int stepOffset, cudaStream_t st) {
    switch (minB) {
    case 1: v1_batch_step_kernel<Rng, 1><<<grid, kCta, 0, st>>>(trials, tiles, nTiles, stepOffset); break;
    case 2: v1_batch_step_kernel<Rng, 2><<<grid, kCta, 0, st>>>(trials, tiles, nTiles, stepOffset); break;
    case 3: v1_batch_step_kernel<Rng, 3><<<grid, kCta, 0, st>>>(trials, tiles, nTiles, stepOffset); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_v1_batch_step(const BatchTrial *trials, const int2 *tiles, const int *nTiles,
                                 int gridTiles, int stepOffset, bool rng, int minB, cudaStream_t st) {
    if (gridTiles <= 0) return cudaSuccess;
    return rng ? launch_batch_variant<true>(minB, trials, tiles, nTiles, gridTiles, stepOffset, st)
               : launch_batch_variant<false>(minB, trials, tiles, nTiles, gridTiles, stepOffset, st);
}

int v1_batch_regs(int minB, bool rng) {
    cudaFuncAttributes a{};
    cudaError_t e = cudaErrorInvalidValue;
    if (rng) {
        if (minB == 1) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<true, 1>);
        if (minB == 2) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<true, 2>);
        if (minB == 3) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<true, 3>);
    } else {
        if (minB == 1) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<false, 1>);
        if (minB == 2) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<false, 2>);
        if (minB == 3) e = cudaFuncGetAttributes(&a, v1_batch_step_kernel<false, 3>);
    }
    return e == cudaSuccess ? a.numRegs : -1;
}

// Per trial: step += the steps it ran in the chunk (K, or fewer at its end), and its FP64
// simulated-time accumulator += those steps * dt.
__global__ void batch_advance_kernel(BatchTrial *trials, int nTrials, int K, double *simTime) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nTrials) return;
    const long long s = *trials[q].step;
    long long k = trials[q].tEnd - s;
    k = k < 0 ? 0 : (k > K ? K : k);
    *trials[q].step = s + k;
    simTime[q] += (double)k * trials[q].dt;
}

cudaError_t launch_batch_advance(BatchTrial *trials, int nTrials, int K, double *simTime, cudaStream_t st) {
    batch_advance_kernel<<<(nTrials + 127) / 128, 128, 0, st>>>(trials, nTrials, K, simTime);
    return cudaGetLastError();
}

// FP64 firing rates of one trial: rate[i] = count[i] / simulated seconds, and the mean over
// its neurons (one CTA, double-precision tree reduction).
__global__ void __launch_bounds__(1024) batch_rates_kernel(const unsigned *counts, int nV1, const double *simTime,
                                                           double *rates, double *meanRate) {
    __shared__ double red[32];
    const double sec = *simTime * 1e-3;
    double acc = 0.0;
    for (int i = threadIdx.x; i < nV1; i += blockDim.x) {
        const double r = sec > 0 ? (double)counts[i] / sec : 0.0;
        if (rates) rates[i] = r;
        acc += r;
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        acc = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (threadIdx.x == 0) *meanRate = acc / (double)nV1;
    }
}

cudaError_t launch_batch_rates(const BatchTrial *, const unsigned *counts, const long long *countOff,
                               const double *simTime, int trial, int nV1, double *rates, double *meanRate,
                               cudaStream_t st) {
    batch_rates_kernel<<<1, 1024, 0, st>>>(counts + countOff[trial], nV1, simTime + trial, rates, meanRate);
    return cudaGetLastError();
}

}  // namespace pv1
