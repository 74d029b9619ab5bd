// Seeding of the per-cell and per-neuron MRG32k3a generators.
//
// Generator `id` of a seed starts 2^76 * id draws after generator 0 (curand_init's sequence
// argument).  curand_init takes one thread about 2.2 ms to get there for any id past 0 (it is a
// serial chain, the same for 512 and 16,384 generators), so only generator 0 is seeded with it
// here; the others are reached with the recurrence's own jump: the state is two vectors of
// three words, one draw multiplies them by A1 mod m1 and A2 mod m2 (P. L'Ecuyer, "Good
// parameters and implementations for combined multiple recursive random number generators",
// Oper. Res. 47, 1999), so id sequences further is a product with A^(2^76 * id), the product of
// the powers A^(2^(76 + k)) over the bits k of id.  Those powers are evaluated by the compiler
// from A by repeated squaring; a thread does one matrix-vector product per set bit.
// Measured on whole runs of the BF16 LGN stage, which seeds its cells each time: 512 cells x 640
// steps 2,376 -> 156 us, 16,384 cells x 16,000 steps 4,718 -> 1,495 us (the seeding kernel was
// 2,245 and 3,250 us of them).
#pragma once

#include <curand_kernel.h>

namespace pv1 {

constexpr unsigned long long kMrgM1 = 4294967296ull - 209ull, kMrgM2 = 4294967296ull - 22853ull;
constexpr int kMrgSpacing = 76;    // log2 of the draws between consecutive sequences
constexpr int kMrgBits = 40;       // sequence numbers below 2^40

struct MrgJump {
    unsigned a1[kMrgBits][9], a2[kMrgBits][9];
};

constexpr MrgJump make_mrg_jump() {
    MrgJump J{};
    // one draw: (s0, s1, s2) -> (s1, s2, a s1 + b s0) and (s1, s2, a s2 + b s0)
    unsigned long long A1[9] = {0, 1, 0, 0, 0, 1, kMrgM1 - 810728ull, 1403580ull, 0};
    unsigned long long A2[9] = {0, 1, 0, 0, 0, 1, kMrgM2 - 1370589ull, 0, 527612ull};
    for (int e = 0; e < kMrgSpacing + kMrgBits; e++) {
        if (e >= kMrgSpacing)
            for (int i = 0; i < 9; i++) {
                J.a1[e - kMrgSpacing][i] = (unsigned)A1[i];
                J.a2[e - kMrgSpacing][i] = (unsigned)A2[i];
            }
        unsigned long long B1[9] = {}, B2[9] = {};
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++)
                for (int k = 0; k < 3; k++) {
                    B1[3 * i + j] = (B1[3 * i + j] + A1[3 * i + k] * A1[3 * k + j] % kMrgM1) % kMrgM1;
                    B2[3 * i + j] = (B2[3 * i + j] + A2[3 * i + k] * A2[3 * k + j] % kMrgM2) % kMrgM2;
                }
        for (int i = 0; i < 9; i++) {
            A1[i] = B1[i];
            A2[i] = B2[i];
        }
    }
    return J;
}

static __constant__ MrgJump kMrgJump = make_mrg_jump();

// Row times vector modulo 2^32 - C: 2^32 = C (mod m), so the high word of each product folds
// into C times itself (three folded products stay below 2^49), once more for the sum, and one
// subtraction ends in [0, m).
template <unsigned C>
__device__ __forceinline__ unsigned mrg_row(const unsigned *a, const unsigned *x) {
    unsigned long long t = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const unsigned long long p = (unsigned long long)a[k] * x[k];
        t += (p >> 32) * C + (p & 0xffffffffull);
    }
    t = (t >> 32) * C + (t & 0xffffffffull);
    constexpr unsigned long long m = 4294967296ull - C;
    return (unsigned)(t >= m ? t - m : t);
}

// curand_init(seed, id, 0, s), bit for bit, for id < 2^40.
__device__ __forceinline__ void mrg_seed(unsigned long long seed, unsigned long long id, curandStateMRG32k3a *s) {
    curand_init(seed, 0ull, 0ull, s);
    unsigned x[3] = {s->s1[0], s->s1[1], s->s1[2]}, y[3] = {s->s2[0], s->s2[1], s->s2[2]};
    for (int k = 0; k < kMrgBits && (id >> k); k++) {
        if (!((id >> k) & 1)) continue;
        unsigned u[3], w[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            u[i] = mrg_row<209u>(kMrgJump.a1[k] + 3 * i, x);
            w[i] = mrg_row<22853u>(kMrgJump.a2[k] + 3 * i, y);
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            x[i] = u[i];
            y[i] = w[i];
        }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        s->s1[i] = x[i];
        s->s2[i] = y[i];
    }
}

// The next uniform of (0, 1], curand_uniform(s) bit for bit: the recurrence and the combination of its two
// parts as published (see the top of the file), in integers.  cuRAND evaluates them in double precision,
// whose rate is a small fraction of single's here.  Measured on the LGN stage of the sweep of 12 trials: the
// sweep 23,376 -> 22,970 us; 16 steps of one block 128.1 -> 126.2 us.
__device__ __forceinline__ float mrg_uniform(curandStateMRG32k3a *s) {
    auto fold = [](unsigned long long a, unsigned long long b, unsigned long long C) {   // a + b mod 2^32 - C
        unsigned long long t = (a >> 32) * C + (a & 0xffffffffull) + (b >> 32) * C + (b & 0xffffffffull);
        t = (t >> 32) * C + (t & 0xffffffffull);
        const unsigned long long m = 4294967296ull - C;
        return (unsigned)(t >= m ? t - m : t);
    };
    const unsigned p1 = fold(1403580ull * s->s1[1], (kMrgM1 - 810728ull) * s->s1[0], 209ull);
    s->s1[0] = s->s1[1];
    s->s1[1] = s->s1[2];
    s->s1[2] = p1;
    const unsigned p2 = fold(527612ull * s->s2[2], (kMrgM2 - 1370589ull) * s->s2[0], 22853ull);
    s->s2[0] = s->s2[1];
    s->s2[1] = s->s2[2];
    s->s2[2] = p2;
    const unsigned z = p1 > p2 ? p1 - p2 : (unsigned)(p1 + kMrgM1 - p2);
    return (float)((double)z * (1.0 / 4294967087.0));   // 1 .. m1 to (0, 1]
}

}  // namespace pv1
