/*
 * Pair production in FP32C evaluated by a whole CTA, one (pair, node) a thread:
 * the float-float form, whose nodes are the longest chain of the FP32C engine
 * and whose pairs are few.
 */
#pragma once

#include "dcs_fp32c.cuh"

namespace noa_dcs {

// Shared memory of a pair-production batch evaluated by (pair, node).
template <int THREADS>
struct Pprod32Smem {
    float pair[sizeof(Pprod32<true>) / sizeof(float)][THREADS];
    float g[8][THREADS], e[8][THREADS];
};

// Evaluates `take` (1 .. THREADS) open pairs with all threads of the CTA, thread
// t < take having pair t in K, q: set up one pair a thread, nodes one (pair,
// node) a thread, each pair's nodes added in order by one thread.  With one
// thread a pair, the 22 or so redo pairs that a CTA has left at the end of a
// call kept it waiting for eight float-float nodes in a row: 1000 / 60013 /
// 250007 pairs of iron 26.7 / 39.8 / 53.4 us, now 16.8 / 29.8 / 43.8 (1e7 pairs
// unchanged); the batched engine with ten elements, which ends a step at each
// element, at 1000 / 1e5 / 1e6 / 1e7 pairs 42.8 / 47.0 / 211 / 1191 -> 34.7 /
// 38.5 / 183 / 1159.  The float form gains less (14.3 / 28.3 / 44.4 us) and loses 6%
// at 1e7 pairs to the round trip through shared memory, so it keeps one thread
// a pair.  Called by every thread; the caller synchronises before the next
// call.
// consts(e) are the constants of pair e's element.
template <bool FINE, int THREADS, typename Consts>
__device__ __forceinline__ double pprod32_batch_mixed(Pprod32Smem<THREADS> &s, int take, double K, double q,
                                                      Consts consts, float &est) {
    constexpr int WORDS = sizeof(Pprod32<FINE>) / sizeof(float);
    const int t = threadIdx.x;
    Pprod32<FINE> p;
    float *w = reinterpret_cast<float *>(&p);
    if (t < take) {
        pprod32_setup<FINE>(K, q, pprod_argmin_ff(K, q, consts(t)), consts(t), p);
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            s.pair[i][t] = w[i];
    }
    __syncthreads();
#pragma unroll 1
    for (int it = t; it < 8 * take; it += THREADS) {
        const int j = it / take, e = it - j * take;
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            w[i] = s.pair[i][e];
        float eg;
        s.g[j][e] = pprod32_node<FINE>(p, j, consts(e), eg);
        s.e[j][e] = eg;
    }
    __syncthreads();
    est = 0.f;
    if (t >= take)
        return 0.;
    KSum I;
    float err = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        I.add(s.g[j][t] * kF8W[j]);
        err += s.e[j][t] * kF8W[j];
    }
    return pprod32_finish(K, q, I, err, consts(t), est);
}

// All pairs of one element.
template <bool FINE, int THREADS>
__device__ __forceinline__ double pprod32_batch(Pprod32Smem<THREADS> &s, int take, double K, double q,
                                                const noa_dcs_consts &c, float &est) {
    return pprod32_batch_mixed<FINE>(s, take, K, q, [&](int) -> const noa_dcs_consts & { return c; }, est);
}

} // namespace noa_dcs
