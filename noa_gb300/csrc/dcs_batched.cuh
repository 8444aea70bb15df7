/*
 * Batched multi-element DCS engine: one persistent launch evaluates one
 * process for up to NOA_DCS_MAX_SEGMENTS elements, each with its own
 * (uneven) number of pairs, stored back to back in K, q and result.
 *
 *  - Work unit: a tile of at most THREADS x items consecutive pairs of one
 *    segment (fewer where the call would not give every CTA a few tiles).
 *    Tiles of all segments form one index space (prefix sums in the
 *    parameters); each CTA takes the next tile from a global counter
 *    (atomicAdd), so CTAs balance across the uneven segments without a
 *    host-side split.  The counter is the engine's only global scratch and is
 *    zeroed by a memset node before each launch.
 *  - Inside a CTA the tile goes through the same compaction as the
 *    single-element kernels: open pairs are appended to a shared-memory work
 *    queue that is popped THREADS at a time (FP64 pair production and
 *    photonuclear: evaluated by the whole CTA, quad_batch); for FP32C, pairs
 *    whose error estimate exceeds the tolerance go to a redo queue evaluated
 *    in FP64 (pair production: evaluated again with its screening log in
 *    float-float arithmetic, and only what that still rejects in FP64).
 *    When the next tile belongs to another segment the queues are drained
 *    first, so every warp evaluates pairs of a single element and the element
 *    constants stay warp-uniform (they are read from the parameter space).
 *  - THREADS is a template parameter (128 or 256), items per thread (1-8) and
 *    CTAs per SM are launch parameters: the autotuner's search space.
 *
 * No counterpart in the reference, which evaluates one element per call.
 */
#pragma once

#include "dcs_fp32c.cuh"
#include "dcs_fp32c_batch.cuh"
#include "dcs_quad.cuh"

#include <atomic>

namespace noa_dcs {

struct BatchParams {
    const double *K;
    const double *q;
    double *out;
    unsigned long long *counter;
    int n_seg;
    int items;
    float tol;
    int tile;  // pairs per tile, at most items x THREADS
    int64_t seg_begin[NOA_DCS_MAX_SEGMENTS + 1];
    int64_t tile_begin[NOA_DCS_MAX_SEGMENTS + 1];
    noa_dcs_consts consts[NOA_DCS_MAX_SEGMENTS];
};

template <int PROC>
__device__ __forceinline__ bool batch_open(double K, double q, const noa_dcs_consts &c) {
    if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_live(K, q, c);
    else if (PROC == NOA_DCS_PROC_PHOTO)
        return photo_live(K, q, c);
    else
        return true;
}

// FP64 of the two processes without a quadrature.
template <int PROC>
__device__ __forceinline__ double batch_eval64(double K, double q, const noa_dcs_consts &c) {
    return PROC == NOA_DCS_PROC_BREMS ? brems_fp64(K, q, c) : ion_fp64(K, q, c);
}

template <int PROC>
__device__ __forceinline__ double batch_eval32(double K, double q, const noa_dcs_consts &c, float &est) {
    if (PROC == NOA_DCS_PROC_BREMS)
        return brems_fp32c(K, q, c, est);
    else if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_fp32c<false>(K, q, c, est);
    else if (PROC == NOA_DCS_PROC_PHOTO)
        return photo_fp32c<false>(K, q, c, est);
    else
        return ion_fp32c(K, q, c, est);
}

__host__ __device__ constexpr bool batch_third_queue(int proc, int prec) {
    return proc == NOA_DCS_PROC_PPROD && prec != NOA_DCS_FP64;
}

// Dynamic shared memory of one CTA: the work queue (items*THREADS + THREADS
// pairs); for FP32C the redo queue (2*THREADS), and for its pair production
// the third queue (2*THREADS) of the pairs its float-float redo step still
// rejects; for the quadrature processes the batch of quad_batch (FP64) or
// quad_redo (FP32C), in the same place as that of pair production's
// float-float step.
template <int THREADS>
struct BatchSmem {
    static constexpr size_t pair_bytes = 2 * sizeof(double) + sizeof(int64_t);
    static __host__ __device__ constexpr size_t queues(int items, int proc, int prec) {
        return pair_bytes * THREADS *
               (items + 1 + (prec != NOA_DCS_FP64 ? 2 : 0) + (batch_third_queue(proc, prec) ? 2 : 0));
    }
    static __host__ __device__ constexpr size_t fine_or_redo() {
        return sizeof(Pprod32Smem<THREADS>) > sizeof(QuadSmem<NOA_DCS_PROC_PPROD, QUAD_REDO>)
                   ? sizeof(Pprod32Smem<THREADS>)
                   : sizeof(QuadSmem<NOA_DCS_PROC_PPROD, QUAD_REDO>);
    }
    static __host__ __device__ constexpr size_t bytes(int items, int proc, int prec) {
        return queues(items, proc, prec) +
               (proc == NOA_DCS_PROC_PPROD
                    ? (prec == NOA_DCS_FP64 ? sizeof(QuadSmem<NOA_DCS_PROC_PPROD, THREADS>)
                                            : fine_or_redo())
                    : 0) +
               (proc == NOA_DCS_PROC_PHOTO
                    ? (prec == NOA_DCS_FP64 ? sizeof(QuadSmem<NOA_DCS_PROC_PHOTO, THREADS>)
                                            : sizeof(QuadSmem<NOA_DCS_PROC_PHOTO, QUAD_REDO>))
                    : 0);
    }
};

// Appends (k, q, i) of the lanes with `push` to a queue (warp-aggregated).
__device__ __forceinline__ void batch_push(bool push, double k, double q, int64_t i, double *QK, double *QQ,
                                           int64_t *QI, int *qn) {
    const unsigned m = __ballot_sync(0xffffffffu, push);
    if (m) {
        const int lane = threadIdx.x & 31;
        int base = 0;
        if (lane == 0)
            base = atomicAdd(qn, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (push) {
            const int pos = base + __popc(m & ((1u << lane) - 1u));
            QK[pos] = k;
            QQ[pos] = q;
            QI[pos] = i;
        }
    }
}

// Pair production, FP32C: evaluates `take` redo-queue entries from `at` with the
// float-float screening log, one (pair, node) a thread; pairs whose estimate
// still exceeds tol go to the third queue (true for this thread's).
template <int THREADS>
__device__ __forceinline__ bool batch_fine_step(Pprod32Smem<THREADS> &s, double *rK, double *rQ, int64_t *rI,
                                                double *xK, double *xQ, int64_t *xI, int *xn, int at, int take,
                                                double *out, const noa_dcs_consts &c, float tol) {
    const int e = at + threadIdx.x;
    const bool valid = (int)threadIdx.x < take;
    bool redo = false;
    double k = 0., q = 0.;
    int64_t i = 0;
    if (valid) {
        k = rK[e];
        q = rQ[e];
        i = rI[e];
    }
    float est;
    const double v = pprod32_batch<true>(s, take, k, q, c, est);
    if (valid) {
        redo = !(est <= tol);
        if (!redo)
            out[i] = v;
    }
    batch_push(redo, k, q, i, xK, xQ, xI, xn);
    return redo;
}

// FP32C: evaluates work-queue entry e (if valid) and writes it or appends it
// to the redo queue.
template <int PROC>
__device__ __forceinline__ bool batch_step32(double *wK, double *wQ, int64_t *wI, double *rK, double *rQ,
                                             int64_t *rI, int *rn, int e, bool valid, double *out,
                                             const noa_dcs_consts &c, float tol) {
    bool redo = false;
    double k = 0., q = 0.;
    int64_t i = 0;
    if (valid) {
        k = wK[e];
        q = wQ[e];
        i = wI[e];
        float est;
        const double v = batch_eval32<PROC>(k, q, c, est);
        redo = !(est <= tol);
        if (!redo)
            out[i] = v;
    }
    batch_push(redo, k, q, i, rK, rQ, rI, rn);
    return redo;
}

template <int PROC, int PREC, int THREADS>
__global__ void __launch_bounds__(THREADS) dcs_batched_kernel(const __grid_constant__ BatchParams p) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int items = p.items;
    const int qcap = items * THREADS + THREADS;
    double *wK = reinterpret_cast<double *>(smem_raw);
    double *wQ = wK + qcap;
    int64_t *wI = reinterpret_cast<int64_t *>(wQ + qcap);
    double *rK = reinterpret_cast<double *>(wI + qcap);
    double *rQ = rK + 2 * THREADS;
    int64_t *rI = reinterpret_cast<int64_t *>(rQ + 2 * THREADS);
    double *xK = reinterpret_cast<double *>(rI + 2 * THREADS);  // third queue (batch_third_queue only)
    double *xQ = xK + 2 * THREADS;
    int64_t *xI = reinterpret_cast<int64_t *>(xQ + 2 * THREADS);
    constexpr bool third = batch_third_queue(PROC, PREC);
    typedef QuadSmem<PROC, PREC == NOA_DCS_FP64 ? THREADS : QUAD_REDO> Quads;
    Quads &quad = *reinterpret_cast<Quads *>(smem_raw + BatchSmem<THREADS>::queues(items, PROC, PREC));
    __shared__ int warp_tot[THREADS / 32];
    __shared__ int tile_open;
    __shared__ int s_rn, s_xn;  // places in the redo queues
    __shared__ unsigned long long s_tile;

    const int tile_size = p.tile;
    const long long total_tiles = p.tile_begin[p.n_seg];
    if (threadIdx.x == 0) {
        s_rn = 0;
        s_xn = 0;
    }
    int qn = 0, rn = 0, xn = 0;  // queue lengths, identical in every thread
    int cur = -1;
    for (;;) {
        if (threadIdx.x == 0)
            s_tile = atomicAdd(p.counter, 1ULL);
        __syncthreads();
        const long long tile = (long long)s_tile;
        __syncthreads();
        const bool done = tile >= total_tiles;
        int seg = cur < 0 ? 0 : cur;
        if (!done) {
            while (seg + 1 < p.n_seg && tile >= p.tile_begin[seg + 1])
                seg++;
            while (seg > 0 && tile < p.tile_begin[seg])
                seg--;
        }
        if (cur >= 0) {
            // Drain the queues of the current element: full batches, or
            // everything when the element changes or the work is done.  One
            // call site each for the step and the redo, so that a pair's result
            // does not depend on where it sits in the queue (nvcc may contract
            // differently in separately inlined copies).
            const bool flush = done || seg != cur;
            const noa_dcs_consts &cc = p.consts[cur];
            // The redo queues' lengths are counted by the barrier that ends a
            // step; each queue is drained below its batch before anything is
            // added to it again (its capacity is a batch and one step's THREADS).
            for (;;) {
                bool did = false, rejected = false;
                if (qn >= THREADS || (flush && qn > 0)) {
                    const int take = qn < THREADS ? qn : THREADS;
                    qn -= take;
                    if constexpr (PREC != NOA_DCS_FP64) {
                        rejected = batch_step32<PROC>(wK, wQ, wI, rK, rQ, rI, &s_rn, qn + threadIdx.x,
                                                      (int)threadIdx.x < take, p.out, cc, p.tol);
                    } else if constexpr (is_quad(PROC)) {
                        quad_batch<PROC, THREADS>(
                            quad, take, cc,
                            [&](int e, double &K, double &q) {
                                K = wK[qn + e];
                                q = wQ[qn + e];
                            },
                            [&](int e, double v) { p.out[wI[qn + e]] = v; });
                    } else if ((int)threadIdx.x < take) {
                        const int e = qn + threadIdx.x;
                        p.out[wI[e]] = batch_eval64<PROC>(wK[e], wQ[e], cc);
                    }
                    did = true;
                }
                if constexpr (PREC == NOA_DCS_FP64) {
                    __syncthreads();
                } else {
                    constexpr int redo_batch = PROC == NOA_DCS_PROC_PHOTO ? QUAD_REDO : THREADS;
                    rn += __syncthreads_count(rejected);
                    while (rn >= redo_batch || (flush && qn == 0 && rn > 0)) {
                        const int take = rn < redo_batch ? rn : redo_batch;
                        rn -= take;
                        if (threadIdx.x == 0)
                            s_rn = rn;
                        if constexpr (third) {
                            rejected = batch_fine_step(*reinterpret_cast<Pprod32Smem<THREADS> *>(&quad), rK, rQ, rI,
                                                       xK, xQ, xI, &s_xn, rn, take, p.out, cc, p.tol);
                            xn += __syncthreads_count(rejected);
                            while (xn >= QUAD_REDO || (flush && qn == 0 && rn == 0 && xn > 0)) {
                                const int some = xn < QUAD_REDO ? xn : QUAD_REDO;
                                xn -= some;
                                if (threadIdx.x == 0)
                                    s_xn = xn;
                                quad_redo<PROC, THREADS>(quad, some, cc, xK + xn, xQ + xn, xI + xn, p.out);
                                __syncthreads();
                            }
                        } else if constexpr (is_quad(PROC)) {
                            quad_redo<PROC, THREADS>(quad, take, cc, rK + rn, rQ + rn, rI + rn, p.out);
                            __syncthreads();
                        } else {
                            if ((int)threadIdx.x < take) {
                                const int e = rn + threadIdx.x;
                                p.out[rI[e]] = PROC == NOA_DCS_PROC_BREMS ? brems_reference(rK[e], rQ[e], cc)
                                                                          : ion_fp64(rK[e], rQ[e], cc);
                            }
                            __syncthreads();
                        }
                        did = true;
                    }
                    if constexpr (third) {
                        // what earlier fine steps left below a batch
                        while (flush && qn == 0 && rn == 0 && xn > 0) {
                            const int some = xn < QUAD_REDO ? xn : QUAD_REDO;
                            xn -= some;
                            if (threadIdx.x == 0)
                                s_xn = xn;
                            quad_redo<PROC, THREADS>(quad, some, cc, xK + xn, xQ + xn, xI + xn, p.out);
                            __syncthreads();
                            did = true;
                        }
                    }
                }
                if (!did)
                    break;
            }
        }
        if (done)
            break;
        cur = seg;
        const noa_dcs_consts &c = p.consts[seg];
        const int64_t seg_end = p.seg_begin[seg + 1];
        const int64_t base = p.seg_begin[seg] + (int64_t)(tile - p.tile_begin[seg]) * tile_size;

        double k[8], r[8];
        unsigned open = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j < items) {
                const int o = j * THREADS + threadIdx.x;
                const int64_t i = base + o;
                if (o < tile_size && i < seg_end) {
                    k[j] = p.K[i];
                    r[j] = p.q[i];
                    if (batch_open<PROC>(k[j], r[j], c))
                        open |= 1u << j;
                    else
                        p.out[i] = 0.;
                }
            }
        }
        int pos = qn + block_scan<THREADS>(__popc(open), warp_tot, &tile_open);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (open & (1u << j)) {
                wK[pos] = k[j];
                wQ[pos] = r[j];
                wI[pos] = base + j * THREADS + threadIdx.x;
                pos++;
            }
        }
        __syncthreads();
        qn += tile_open;
    }
}

// Raises a kernel's dynamic shared-memory limit once per device to the most
// it can take (the device's opt-in maximum less the kernel's static shared
// memory; `done` is the kernel's own flag table), so that only the first
// launch on a device above 48 KB sets a function attribute and later
// launches, including launches inside a caller's stream capture, set none.
constexpr int kSmemOptinDevices = 64;
template <typename Kernel>
inline cudaError_t smem_optin_once(Kernel k, size_t smem, std::atomic<bool> (&done)[kSmemOptinDevices]) {
    if (smem <= 48 * 1024)
        return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev >= 0 && dev < kSmemOptinDevices && done[dev].load(std::memory_order_acquire))
        return cudaSuccess;
    int optin = 0;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess)
        return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, k);
    if (e != cudaSuccess)
        return e;
    const int max_dynamic = optin - (int)fa.sharedSizeBytes;
    if (max_dynamic <= 0 || smem > (size_t)max_dynamic)
        return cudaErrorInvalidValue;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dynamic);
    if (e == cudaSuccess && dev >= 0 && dev < kSmemOptinDevices)
        done[dev].store(true, std::memory_order_release);
    return e;
}

} // namespace noa_dcs
