/*
 * FP64 muon DCS kernels for sm_103a.
 *
 * Two launch shapes:
 *
 *  - map kernel (bremsstrahlung, ionisation): every pair is live or nearly so
 *    and the body is short: one pair a thread and step.
 *
 *  - compacting kernel (pair production, photonuclear): ~46% / ~80% of the
 *    pairs of the seeded workload are closed kinematically and the live ones
 *    run an 8- or 9-node quadrature.  A CTA classifies a tile with the cheap
 *    bound checks (the reference's early returns), writes the zeros straight
 *    away, and appends the live pairs (K, q, index) to a queue in shared
 *    memory.  Whenever the queue holds a full batch, and at the end for the
 *    remainder, the CTA evaluates it together (quad_batch).  The tile follows
 *    the size of the call, so that a short list spreads over the SMs.  No
 *    global scratch.
 *
 * Each kernel calls the evaluation from exactly one place.  nvcc inlines
 * every call site separately and may contract a * b + c into an FMA
 * differently in each copy, so two call sites (a full-batch drain and a tail,
 * or an unrolled item loop) could round the same pair differently depending
 * on where it sits in the queue.  With one call site a pair's result depends
 * on (K, q) only.
 *
 * The reference launches one thread per pair on the legacy stream
 * (common.cuh:33-56) and recomputes three pow() per bremsstrahlung evaluation
 * (physics.hh:126-128); it has no GPU pair-production, photonuclear or
 * ionisation kernel.
 */
#include "dcs_quad.cuh"

#include <cuda_runtime.h>

namespace noa_dcs {

constexpr int MAP_THREADS = 128;
constexpr int MAP_MIN_CTAS = 10;
// One pair a thread up to 1000 CTAs an SM (19e6 pairs), grid-stride beyond:
// the hardware's own distribution of short CTAs balances the SMs better than
// a resident grid (1e7 pairs 516 / 360 us against 525 / 368 us at 10 CTAs an
// SM, 1e6 pairs 69 / 52 against 72 / 53).
constexpr int MAP_GRID_CTAS = 1000;
constexpr int CMP_THREADS = 128;
constexpr int CMP_ITEMS = 1;  // 2 items' queue takes the shared memory of the last resident CTA: 1% slower
constexpr int CMP_TILE = CMP_THREADS * CMP_ITEMS;  // largest tile
constexpr int CMP_QCAP = CMP_TILE + CMP_THREADS;

// Resident CTAs per SM that the compacting kernels are compiled for (the
// register budget per thread follows) and their grid is made of.  Measured at
// 1e7 pairs: pair production 3.44 / 3.34 / 3.36 ms at 5 / 6 / 7; photonuclear
// 1.96 / 1.94 / 1.92 ms at 6 / 7 / 8 (the most that shared memory holds).
#ifndef NOA_DCS_PPROD_MIN_CTAS
#define NOA_DCS_PPROD_MIN_CTAS 6
#endif
#ifndef NOA_DCS_PHOTO_MIN_CTAS
#define NOA_DCS_PHOTO_MIN_CTAS 8
#endif
template <int PROC>
constexpr int cmp_min_ctas() {
    return PROC == NOA_DCS_PROC_PHOTO ? NOA_DCS_PHOTO_MIN_CTAS : NOA_DCS_PPROD_MIN_CTAS;
}

template <int PROC>
__device__ __forceinline__ bool live_fp64(double K, double q, const noa_dcs_consts &c) {
    if (PROC == NOA_DCS_PROC_PPROD)
        return pprod_live(K, q, c);
    else
        return photo_live(K, q, c);
}

template <int PROC>
__global__ void __launch_bounds__(MAP_THREADS, MAP_MIN_CTAS) dcs_fp64_map_kernel(const double *__restrict__ K,
                                                                   const double *__restrict__ q, double *out,
                                                                   int64_t n, const noa_dcs_consts c) {
#pragma unroll 1  // one inlined copy of the evaluation
    for (int64_t i = (int64_t)blockIdx.x * MAP_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * MAP_THREADS)
        out[i] = PROC == NOA_DCS_PROC_BREMS ? brems_fp64(K[i], q[i], c) : ion_fp64(K[i], q[i], c);
}

template <int PROC>
__global__ void __launch_bounds__(CMP_THREADS, cmp_min_ctas<PROC>())
    dcs_fp64_compact_kernel(const double *__restrict__ K, const double *__restrict__ q, double *out, int64_t n, int tile,
                            const noa_dcs_consts c) {
    __shared__ double qK[CMP_QCAP];
    __shared__ double qQ[CMP_QCAP];
    __shared__ int64_t qI[CMP_QCAP];
    __shared__ QuadSmem<PROC, CMP_THREADS> quad;
    __shared__ int warp_tot[CMP_THREADS / 32];
    __shared__ int tile_live;
    int qn = 0; // queue length, identical in every thread
    int64_t base = (int64_t)blockIdx.x * tile;
    for (;;) {
        const bool more = base < n;  // block-uniform
        if (more) {
            double k[CMP_ITEMS], r[CMP_ITEMS];
            unsigned live = 0;
#pragma unroll
            for (int j = 0; j < CMP_ITEMS; j++) {
                const int o = j * CMP_THREADS + threadIdx.x;
                const int64_t i = base + o;
                if (o < tile && i < n) {
                    k[j] = K[i];
                    r[j] = q[i];
                    if (live_fp64<PROC>(k[j], r[j], c))
                        live |= 1u << j;
                    else
                        out[i] = 0.;
                }
            }
            int pos = qn + block_scan<CMP_THREADS>(__popc(live), warp_tot, &tile_live);
#pragma unroll
            for (int j = 0; j < CMP_ITEMS; j++) {
                if (live & (1u << j)) {
                    qK[pos] = k[j];
                    qQ[pos] = r[j];
                    qI[pos] = base + j * CMP_THREADS + threadIdx.x;
                    pos++;
                }
            }
            __syncthreads();
            qn += tile_live;
            base += (int64_t)gridDim.x * tile;
        }
        // full batches while tiles remain, then the remainder: one call site
        while (qn >= CMP_THREADS || (!more && qn > 0)) {
            const int take = qn < CMP_THREADS ? qn : CMP_THREADS;
            const int first = qn - take;
            quad_batch<PROC, CMP_THREADS>(
                quad, take, c,
                [&](int e, double &k, double &r) {
                    k = qK[first + e];
                    r = qQ[first + e];
                },
                [&](int e, double v) { out[qI[first + e]] = v; });
            qn -= take;
            __syncthreads();
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

static int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

template <int PROC>
static cudaError_t launch_map(const double *K, const double *q, double *out, int64_t n, const noa_dcs_consts &c,
                              cudaStream_t s) {
    const int64_t blocks = ceil_div(n, MAP_THREADS);
    const int64_t cap = (int64_t)sm_count() * MAP_GRID_CTAS;
    dcs_fp64_map_kernel<PROC><<<(int)(blocks < cap ? blocks : cap), MAP_THREADS, 0, s>>>(K, q, out, n, c);
    return cudaGetLastError();
}

// One resident wave at most, in equal tiles: the largest tile while the call
// fills it, else n spread over all resident CTAs, so that a short list reaches
// every SM; not below 8 pairs (two warps of nodes).
template <int PROC>
static cudaError_t launch_compact(const double *K, const double *q, double *out, int64_t n,
                                  const noa_dcs_consts &c, cudaStream_t s) {
    const int64_t cap = (int64_t)sm_count() * cmp_min_ctas<PROC>();
    const int64_t steps = ceil_div(n, cap * CMP_TILE);
    int64_t tile = ceil_div(n, cap * steps);
    tile = tile < 8 ? 8 : tile;
    dcs_fp64_compact_kernel<PROC><<<(int)ceil_div(n, tile * steps), CMP_THREADS, 0, s>>>(K, q, out, n, (int)tile, c);
    return cudaGetLastError();
}

} // namespace noa_dcs

using namespace noa_dcs;

cudaError_t noa_dcs_launch_fp64(int process, const double *K, const double *q, double *out, int64_t n,
                                const noa_dcs_consts *c, cudaStream_t stream) {
    if (n <= 0)
        return cudaSuccess;
    switch (process) {
    case NOA_DCS_PROC_BREMS:
        return launch_map<NOA_DCS_PROC_BREMS>(K, q, out, n, *c, stream);
    case NOA_DCS_PROC_PPROD:
        return launch_compact<NOA_DCS_PROC_PPROD>(K, q, out, n, *c, stream);
    case NOA_DCS_PROC_PHOTO:
        return launch_compact<NOA_DCS_PROC_PHOTO>(K, q, out, n, *c, stream);
    case NOA_DCS_PROC_ION:
        return launch_map<NOA_DCS_PROC_ION>(K, q, out, n, *c, stream);
    default:
        return cudaErrorInvalidValue;
    }
}
