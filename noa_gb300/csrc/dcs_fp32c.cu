/*
 * FP32-compensated DCS kernels (precision NOA_DCS_FP32C) for sm_103a.
 *
 * Pair production and photonuclear use the compacting kernel of the FP64 path
 * (dcs_fp64.cu) with a second queue:
 *
 *   1. a CTA classifies a tile of 32 to 1024 pairs with the exact kinematic
 *      bounds, writes the zeros, and appends the open pairs to the shared-memory work
 *      queue;
 *   2. whenever the work queue holds 256 pairs, each thread pops one and
 *      evaluates it in FP32 (dcs_fp32c.cuh), which also returns an estimate
 *      of its relative error; results within `tol` are written, the others
 *      are appended (warp-aggregated) to a shared-memory redo queue;
 *   3. the redo queue is evaluated in FP64 by quad_redo (photonuclear), or
 *      (pair production) again in FP32, 256 pairs at a time and one (pair,
 *      node) a thread, with the screening log in float-float arithmetic
 *      (pprod32_batch); the ~1% of those still above `tol` go to a third
 *      queue, evaluated in FP64 by quad_redo.
 *
 * Bremsstrahlung and ionisation are evaluated for every pair, so they have no
 * work queue: a thread evaluates the pairs it loads, and the rejected ones go
 * through a redo queue, 256 at a time.  With the work queue, 1e7 pairs of iron
 * took 138 / 144 us (barriers were the largest stall), now 107 / 118; 61 pairs
 * 3.7 / 3.2 us, now 2.1 / 2.4.
 *
 * The tile follows the size of the call, so that a short list spreads over
 * the SMs.
 *
 * FP64 work is thus proportional to the redo fraction (0-0.5% of open pairs
 * at tol = 1e-6), and every warp of every phase runs with all lanes busy.
 * No global scratch.
 */
#include "dcs_fp32c.cuh"
#include "dcs_fp32c_batch.cuh"
#include "dcs_quad.cuh"

#include <cuda_runtime.h>

namespace noa_dcs {

constexpr int F_THREADS = 256;
constexpr int F_ITEMS = 4;
constexpr int F_TILE = F_THREADS * F_ITEMS;
constexpr int F_QCAP = F_TILE + F_THREADS;
constexpr int F_RCAP = 2 * F_THREADS;

// Resident CTAs per SM that each kernel is compiled for (its register budget
// follows) and its grid is made of.  Measured at 1e7 pairs: pair production
// 1.21 ms at 2, 1.17 at 3 and 1.19 at 4 (with half the tile, for the shared
// memory), but 63 us against 72 and 69 at 250007; photonuclear 463 us at 4
// (64 registers, spilling), 445 at 3, 460 at 5; bremsstrahlung / ionisation
// with their pairs through a work queue 136 / 142 us at 4, 141 / 148 at 3,
// 144 / 146 at 5.  (Since then 12% fewer instructions: pair production 1.07 ms,
// photonuclear 438 us.)
template <int PROC>
constexpr int f32_min_ctas() {
    return PROC == NOA_DCS_PROC_PPROD ? 2 : (PROC == NOA_DCS_PROC_PHOTO ? 3 : 4);
}

template <int PROC>
__device__ __forceinline__ double eval32(double K, double q, const noa_dcs_consts &c, float &est) {
    if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_fp32c<false>(K, q, c, est);
    else
        return photo_fp32c<false>(K, q, c, est);
}

template <int PROC>
__device__ __forceinline__ bool open32(double K, double q, const noa_dcs_consts &c) {
    if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_live(K, q, c);
    else
        return photo_live(K, q, c);
}

// Pair production's float-float step.
template <int PROC>
struct FineSmem {};
template <>
struct FineSmem<NOA_DCS_PROC_PPROD> : Pprod32Smem<F_THREADS> {};

// The third queue exists for pair production only.
template <int PROC>
constexpr int f32_xcap() {
    return PROC == NOA_DCS_PROC_PPROD ? F_THREADS + QUAD_REDO : 1;
}

template <int PROC>
struct Queues {
    double wK[F_QCAP], wQ[F_QCAP];
    int64_t wI[F_QCAP];
    double rK[F_RCAP], rQ[F_RCAP];
    int64_t rI[F_RCAP];
    double xK[f32_xcap<PROC>()], xQ[f32_xcap<PROC>()];
    int64_t xI[f32_xcap<PROC>()];
    QuadSmem<PROC, QUAD_REDO> quad;
    FineSmem<PROC> fine;
    int warp_tot[F_THREADS / 32];
    int tile_open;
    int rn, xn;
};

// Appends (k, q, i) of the lanes with `push` to a queue (warp-aggregated).
__device__ __forceinline__ void push_queue(bool push, double k, double q, int64_t i, double *QK, double *QQ,
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

// Evaluates work-queue entry e (if valid) in FP32 and appends it to the redo
// queue when its error estimate exceeds tol (and returns that).
template <int PROC>
__device__ __forceinline__ bool fp32_step(Queues<PROC> &s, int at, int take, double *out, const noa_dcs_consts &c,
                                          float tol) {
    const int e = at + threadIdx.x;
    const bool valid = (int)threadIdx.x < take;
    bool redo = false;
    double k = 0., q = 0.;
    int64_t i = 0;
    if (valid) {
        k = s.wK[e];
        q = s.wQ[e];
        i = s.wI[e];
        float est;
        const double v = eval32<PROC>(k, q, c, est);
        redo = !(est <= tol);
        if (!redo)
            out[i] = v;
    }
    push_queue(redo, k, q, i, s.rK, s.rQ, s.rI, &s.rn);
    return redo;
}

// Pair production: evaluates `take` redo-queue entries from `at` with the
// float-float screening log and appends to the third queue those whose
// estimate still exceeds tol (true for this thread's).
template <int PROC>
__device__ __forceinline__ bool fine_step(Queues<PROC> &s, int at, int take, double *out, const noa_dcs_consts &c,
                                          float tol) {
    const int e = at + threadIdx.x;
    const bool valid = (int)threadIdx.x < take;
    bool redo = false;
    double k = 0., q = 0.;
    int64_t i = 0;
    if (valid) {
        k = s.rK[e];
        q = s.rQ[e];
        i = s.rI[e];
    }
    float est;
    const double v = pprod32_batch<true>(s.fine, take, k, q, c, est);
    if (valid) {
        redo = !(est <= tol);
        if (!redo)
            out[i] = v;
    }
    push_queue(redo, k, q, i, s.xK, s.xQ, s.xI, &s.xn);
    return redo;
}

// Bremsstrahlung and ionisation: every pair is evaluated where it was loaded,
// and only the rejected ones (0.3 - 0.6% and less) go through a queue, which
// holds what is left of a batch and one tile of which every pair is rejected.
struct RedoQueue {
    double K[F_THREADS + F_TILE], Q[F_THREADS + F_TILE];
    int64_t I[F_THREADS + F_TILE];
    int n;
};

template <int PROC>
__global__ void __launch_bounds__(F_THREADS, f32_min_ctas<PROC>()) dcs_fp32c_map_kernel(
    const double *__restrict__ K, const double *__restrict__ q, double *out, int64_t n, int tile,
    const __grid_constant__ noa_dcs_consts c, float tol) {
    static_assert(!is_quad(PROC), "the quadrature processes compact their open pairs");
    __shared__ RedoQueue s;
    if (threadIdx.x == 0)
        s.n = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * tile;
    for (int64_t base = (int64_t)blockIdx.x * tile; base < n; base += stride) {
        const int here = n - base < tile ? (int)(n - base) : tile;
        int o = threadIdx.x;
        double k_next = 1., r_next = 1.;
        if (o < here) {
            k_next = K[base + o];
            r_next = q[base + o];
        }
        // one call site of the evaluation, the next pair requested before it
#pragma unroll 1
        for (int first = 0; first < here; first += F_THREADS, o += F_THREADS) {
            const double k = k_next, r = r_next;
            if (o + F_THREADS < here) {
                k_next = K[base + o + F_THREADS];
                r_next = q[base + o + F_THREADS];
            }
            bool redo = false;
            if (o < here) {
                float est;
                const double v = PROC == NOA_DCS_PROC_BREMS ? brems_fp32c(k, r, c, est) : ion_fp32c(k, r, c, est);
                redo = !(est <= tol);
                if (!redo)
                    out[base + o] = v;
            }
            push_queue(redo, k, r, base + o, s.K, s.Q, s.I, &s.n);
        }
        // All of this tile's entries are in; the second barrier keeps the next
        // tile's (and the drain's new length) behind every thread's reading.
        __syncthreads();
        int rn = s.n;
        __syncthreads();
        const bool last = base + stride >= n;
        while (rn >= F_THREADS || (last && rn > 0)) {
            const int take = rn < F_THREADS ? rn : F_THREADS;
            rn -= take;
            if (threadIdx.x == 0)
                s.n = rn;
            if ((int)threadIdx.x < take) {
                const int e = rn + threadIdx.x;
                // bremsstrahlung's redo pairs are those at the edge
                out[s.I[e]] = PROC == NOA_DCS_PROC_BREMS ? brems_reference(s.K[e], s.Q[e], c)
                                                         : ion_fp64(s.K[e], s.Q[e], c);
            }
            __syncthreads();
        }
    }
}

// Pair production and photonuclear.
template <int PROC>
__global__ void __launch_bounds__(F_THREADS, f32_min_ctas<PROC>()) dcs_fp32c_kernel(const double *__restrict__ K,
                                                              const double *__restrict__ q, double *out, int64_t n,
                                                              int tile, const __grid_constant__ noa_dcs_consts c,
                                                              float tol) {
    __shared__ Queues<PROC> s;
    if (threadIdx.x == 0) {
        s.rn = 0;
        s.xn = 0;
    }
    int qn = 0, rn = 0, xn = 0;
    int64_t base = (int64_t)blockIdx.x * tile;
    for (;;) {
        const bool more = base < n;  // block-uniform
        if (more) {
            double k[F_ITEMS], r[F_ITEMS];
            unsigned open = 0;
#pragma unroll
            for (int j = 0; j < F_ITEMS; j++) {
                const int o = j * F_THREADS + threadIdx.x;
                const int64_t i = base + o;
                if (o < tile && i < n) {
                    k[j] = K[i];
                    r[j] = q[i];
                    if (open32<PROC>(k[j], r[j], c))
                        open |= 1u << j;
                    else
                        out[i] = 0.;
                }
            }
            int pos = qn + block_scan<F_THREADS>(__popc(open), s.warp_tot, &s.tile_open);
#pragma unroll
            for (int j = 0; j < F_ITEMS; j++) {
                if (open & (1u << j)) {
                    s.wK[pos] = k[j];
                    s.wQ[pos] = r[j];
                    s.wI[pos] = base + j * F_THREADS + threadIdx.x;
                    pos++;
                }
            }
            __syncthreads();
            qn += s.tile_open;
            base += (int64_t)gridDim.x * tile;
        }
        // One call site each for the FP32 step, the redo step and the FP64
        // evaluation (see the FP64 kernels): full batches while tiles remain,
        // everything at the end.
        // The lengths of the redo queues are counted by the barrier that ends a
        // step, identical in every thread; the shared counters only hand out
        // places.  Each queue is drained below its batch before anything is
        // added to it again, so that its capacity (a batch and one step's 256)
        // holds even when every pair is rejected.
        for (;;) {
            bool did = false, rejected = false;
            if (qn >= F_THREADS || (!more && qn > 0)) {
                const int take = qn < F_THREADS ? qn : F_THREADS;
                rejected = fp32_step<PROC>(s, qn - take, take, out, c, tol);
                qn -= take;
                did = true;
            }
            rn += __syncthreads_count(rejected);
            constexpr int redo_batch = PROC == NOA_DCS_PROC_PHOTO ? QUAD_REDO : F_THREADS;
            while (rn >= redo_batch || (!more && qn == 0 && rn > 0)) {
                const int take = rn < redo_batch ? rn : redo_batch;
                rn -= take;
                if (threadIdx.x == 0)
                    s.rn = rn;
                if constexpr (PROC == NOA_DCS_PROC_PPROD) {
                    rejected = fine_step<PROC>(s, rn, take, out, c, tol);
                    xn += __syncthreads_count(rejected);
                    while (xn >= QUAD_REDO || (!more && qn == 0 && rn == 0 && xn > 0)) {
                        const int some = xn < QUAD_REDO ? xn : QUAD_REDO;
                        xn -= some;
                        if (threadIdx.x == 0)
                            s.xn = xn;
                        quad_redo<PROC, F_THREADS>(s.quad, some, c, s.xK + xn, s.xQ + xn, s.xI + xn, out);
                        __syncthreads();
                    }
                } else {
                    quad_redo<PROC, F_THREADS>(s.quad, take, c, s.rK + rn, s.rQ + rn, s.rI + rn, out);
                    __syncthreads();
                }
                did = true;
            }
            if constexpr (PROC == NOA_DCS_PROC_PPROD) {
                // what earlier fine steps left below a batch
                while (!more && qn == 0 && rn == 0 && xn > 0) {
                    const int some = xn < QUAD_REDO ? xn : QUAD_REDO;
                    xn -= some;
                    if (threadIdx.x == 0)
                        s.xn = xn;
                    quad_redo<PROC, F_THREADS>(s.quad, some, c, s.xK + xn, s.xQ + xn, s.xI + xn, out);
                    __syncthreads();
                    did = true;
                }
            }
            if (!did)
                break;
        }
        if (!more)
            break;
    }
}

static int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

template <int PROC>
static cudaError_t launch(const double *K, const double *q, double *out, int64_t n, const noa_dcs_consts &c,
                          float tol, cudaStream_t s) {
    // One resident wave at most, in equal tiles: the largest tile while the
    // call fills it, else n spread over all resident CTAs (a warp at least).
    // Equal tiles of any length beat multiples of 32, 64 or 256 (1e7 pairs:
    // bremsstrahlung 140 us against 143, 147 and 148).
    const int64_t cap = (int64_t)sm_count() * f32_min_ctas<PROC>();
    const int64_t steps = (n + cap * F_TILE - 1) / (cap * F_TILE);
    int64_t tile = (n + cap * steps - 1) / (cap * steps);
    tile = tile < 32 ? 32 : tile;
    const int grid = (int)((n + tile * steps - 1) / (tile * steps));
    if constexpr (is_quad(PROC))
        dcs_fp32c_kernel<PROC><<<grid, F_THREADS, 0, s>>>(K, q, out, n, (int)tile, c, tol);
    else
        dcs_fp32c_map_kernel<PROC><<<grid, F_THREADS, 0, s>>>(K, q, out, n, (int)tile, c, tol);
    return cudaGetLastError();
}

} // namespace noa_dcs

using namespace noa_dcs;

cudaError_t noa_dcs_launch_fp32c(int process, const double *K, const double *q, double *out, int64_t n,
                                 const noa_dcs_consts *c, float tol, cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    switch (process) {
    case NOA_DCS_PROC_BREMS:
        return launch<NOA_DCS_PROC_BREMS>(K, q, out, n, *c, tol, stream);
    case NOA_DCS_PROC_PPROD:
        return launch<NOA_DCS_PROC_PPROD>(K, q, out, n, *c, tol, stream);
    case NOA_DCS_PROC_PHOTO:
        return launch<NOA_DCS_PROC_PHOTO>(K, q, out, n, *c, tol, stream);
    case NOA_DCS_PROC_ION:
        return launch<NOA_DCS_PROC_ION>(K, q, out, n, *c, tol, stream);
    default:
        return cudaErrorInvalidValue;
    }
}
