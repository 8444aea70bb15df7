/*
 * The two quadrature processes (pair production, 8 nodes; photonuclear, 9)
 * evaluated by a whole CTA: a batch of queued pairs is set up one pair a
 * thread, its nodes are evaluated one (pair, node) a thread, and each pair's
 * node values are summed in node order by one thread.
 *
 * Against one thread a pair with its nodes in sequence this fills a CTA
 * however few pairs a batch holds: a node is a chain of 14 - 24 elementary
 * functions (about 4 us of latency), so a short list of pairs, a tile's
 * remainder or a table with one kinetic energy per CTA waited for 8 or 9 of
 * them.  The node constants of a pair go through shared memory, which also
 * takes them out of the registers of the node loop.  Full batches do the
 * same work as before (node r of pair t in round r).
 *
 * One call site each of setup, node and finish: nvcc may contract separately
 * inlined copies differently, and a pair's result must not depend on its
 * place in a batch.
 */
#pragma once

#include "dcs_fp64.cuh"
#include "dcs_launch.h"

namespace noa_dcs {

template <int PROC>
struct Quad;

template <>
struct Quad<NOA_DCS_PROC_PPROD> {
    static constexpr int NODES = 8;
    typedef PprodPair Pair;
    static __device__ __forceinline__ void setup(double K, double q, const noa_dcs_consts &c, Pair &p) {
        pprod_setup(K, q, c, p);
    }
    static __device__ __forceinline__ double node(const Pair &p, int j, const noa_dcs_consts &c) {
        return pprod_node(p, j, c);
    }
    static __device__ __forceinline__ double weight(int j) { return kGL8W[j]; }
    static __device__ __forceinline__ double finish(double K, double q, const Pair &p, double sum,
                                                    const noa_dcs_consts &c) {
        return pprod_finish(K, q, p.tmin, sum, c);
    }
};

template <>
struct Quad<NOA_DCS_PROC_PHOTO> {
    static constexpr int NODES = 9;
    typedef PhotoPair Pair;
    static __device__ __forceinline__ void setup(double K, double q, const noa_dcs_consts &c, Pair &p) {
        photo_setup(K, q, c, p);
    }
    static __device__ __forceinline__ double node(const Pair &p, int j, const noa_dcs_consts &c) {
        return photo_node(p, j, c);
    }
    static __device__ __forceinline__ double weight(int j) { return kGL9W[j]; }
    static __device__ __forceinline__ double finish(double K, double q, const Pair &p, double sum,
                                                    const noa_dcs_consts &c) {
        return photo_finish(K, q, p.hd, sum, c);
    }
};

__host__ __device__ constexpr bool is_quad(int proc) {
    return proc == NOA_DCS_PROC_PPROD || proc == NOA_DCS_PROC_PHOTO;
}

// Shared memory of a batch of at most B pairs.
template <int PROC, int B>
struct QuadSmem {
    static constexpr int WORDS = sizeof(typename Quad<PROC>::Pair) / sizeof(double);
    double pair[WORDS][B];
    double val[Quad<PROC>::NODES][B];
};
template <int B>
struct QuadSmem<NOA_DCS_PROC_BREMS, B> {};
template <int B>
struct QuadSmem<NOA_DCS_PROC_ION, B> {};

// Evaluates `take` (1 .. B) open pairs with all threads of the CTA: load(e, K,
// q) gives pair e, store(e, dcs) takes its value, both called by one thread
// per pair; consts(e) are the constants of pair e's element.  Called by every thread; starts and ends with work that only its
// own pairs' threads see, so the caller synchronises before it changes what
// load reads and before it reuses the shared memory.
template <int PROC, int THREADS, int B, typename Consts, typename Load, typename Store>
__device__ __forceinline__ void quad_batch_mixed(QuadSmem<PROC, B> &s, int take, Consts consts, Load load,
                                                 Store store) {
    typedef Quad<PROC> Q;
    typedef QuadSmem<PROC, B> S;
    static_assert(B <= THREADS, "one thread per pair");
    const int t = threadIdx.x;
    double K = 1., q = 1.;
    if (t < take) {
        load(t, K, q);
        typename Q::Pair p;
        Q::setup(K, q, consts(t), p);
        const double *w = reinterpret_cast<const double *>(&p);
#pragma unroll
        for (int i = 0; i < S::WORDS; i++)
            s.pair[i][t] = w[i];
    }
    __syncthreads();
    const int items = take * Q::NODES;
#pragma unroll 1
    for (int it = t; it < items; it += THREADS) {
        const int j = it / take, e = it - j * take;
        typename Q::Pair p;
        double *w = reinterpret_cast<double *>(&p);
#pragma unroll
        for (int i = 0; i < S::WORDS; i++)
            w[i] = s.pair[i][e];
        s.val[j][e] = Q::node(p, j, consts(e));
    }
    __syncthreads();
    if (t < take) {
        typename Q::Pair p;
        double *w = reinterpret_cast<double *>(&p);
#pragma unroll
        for (int i = 0; i < S::WORDS; i++)
            w[i] = s.pair[i][t];
        double sum = 0.;
#pragma unroll
        for (int j = 0; j < Q::NODES; j++)
            sum = fma(Q::weight(j), s.val[j][t], sum);
        store(t, Q::finish(K, q, p, sum, consts(t)));
    }
}

// All pairs of one element.
template <int PROC, int THREADS, int B, typename Load, typename Store>
__device__ __forceinline__ void quad_batch(QuadSmem<PROC, B> &s, int take, const noa_dcs_consts &c, Load load,
                                           Store store) {
    quad_batch_mixed<PROC, THREADS>(s, take, [&](int) -> const noa_dcs_consts & { return c; }, load, store);
}

// FP64 redo of the FP32C kernels: `take` (1 .. QUAD_REDO) pairs of a queue
// into out[I].  Out of line, so that the rare FP64 path does not set the
// kernel's register budget; 32 pairs at a time, whose nodes are one round of
// 256 threads (one thread a pair ran its 8 nodes for 60 us at the end of a
// call, for a handful of pairs).
constexpr int QUAD_REDO = 32;
template <int PROC, int THREADS>
static __device__ __noinline__ void quad_redo(QuadSmem<PROC, QUAD_REDO> &s, int take, const noa_dcs_consts &c,
                                              const double *qK, const double *qQ, const int64_t *qI, double *out) {
    quad_batch<PROC, THREADS>(
        s, take, c,
        [&](int e, double &K, double &q) {
            K = qK[e];
            q = qQ[e];
        },
        [&](int e, double v) { out[qI[e]] = v; });
}

// Exclusive scan of one small count per thread over the CTA; `total` takes
// the sum.  Two barriers.
template <int THREADS>
__device__ __forceinline__ int block_scan(int v, int *warp_tot, int *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int w = lane < (THREADS >> 5) ? warp_tot[lane] : 0;
        int s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o)
                s += y;
        }
        if (lane < (THREADS >> 5))
            warp_tot[lane] = s - w;
        if (lane == 31)
            *total = s;
    }
    __syncthreads();
    return warp_tot[warp] + x - v;
}

} // namespace noa_dcs
