/*
 * Learned DCS surrogate: training-data preparation, forward / backward / Adam
 * kernels and the C ABI of the model object (include/noa_dcs.h,
 * noa_dcs_mlp_*).  No counterpart in the reference.
 *
 * Training runs on the 5th-generation tensor cores (tcgen05.mma, operands in
 * shared memory, FP32 accumulators in TMEM; tcgen05.cuh) in BF16 with FP32
 * accumulation: the 128 x 128 products of the two hidden layers, their input
 * gradients and their weight gradients.  The first layer (4 inputs) and
 * the output layer (1 output) are FP32 on the CUDA cores.  In the forward
 * products both the hidden activations and the weights enter as a BF16 hi +
 * lo pair (x = hi + lo, 16 significant bits), as three products
 * A_hi W_hi + A_lo W_hi + A_hi W_lo with FP32 accumulation; the weight pairs
 * are refreshed from the FP32 master copy after every Adam step, so training
 * sees the numerics of inference.  Gradients flow in single BF16.
 *
 * One kernel takes a tile of 128 samples through the whole network and back
 * (mlp_tile_kernel); a training step is that kernel and Adam.  A kernel per
 * product, with every activation and gradient through global memory, took 15
 * launches and 180 us a step at batch 8192, most of it staging, launch latency
 * and 8192 atomics on the loss.
 *
 * Loss: mean squared error of the normalised residual (mlp.cuh).
 */
#include "dcs_fp64.cuh"
#include "dcs_launch.h"
#include "mlp.cuh"
#include "tcgen05.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <initializer_list>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>

using namespace noa_mlp;

namespace {

constexpr int NPARAM_PAD = (NPARAM + 3) & ~3;  // parameter-sized buffers, padded to 16 bytes
constexpr int TILE_THREADS = 512;
using noa_tc::MAT_BYTES;

// Transposed operands (rows = units, K = samples) are written by threads that
// own a sample: K-adjacent core matrices lie 144 bytes apart instead of 128,
// so that the 32 samples of a warp reach different banks.
constexpr uint32_t T_LBO = 144, T_SBO = 16 * T_LBO, T_BYTES = 16 * T_SBO;

// Dynamic shared memory: six 128 x 128 BF16 operands, the last with room for a
// transposed one, and 1 KB of alignment slack.
constexpr size_t TILE_SMEM = 5 * MAT_BYTES + T_BYTES + 1024;

struct TileArgs {
    const float *X;         // [.][4] normalised features
    const float *T;         // [.] targets (training)
    const int32_t *perm;    // sample of row i, or nullptr: i itself
    const float *P;         // parameters
    const __nv_bfloat16 *Wb;  // six 128 x 128 matrices, see mlp_round_weights_kernel
    float *G;               // gradient, accumulated (training)
    float *loss;            // accumulated (training)
    float *pred;            // predictions (not training)
    unsigned int *status;   // set to NOA_DCS_ERROR_TIMEOUT if an mbarrier wait expires
    float inv_batch;
    int M;
};

// 8 FP32 values -> 8 BF16 (hi), and the rounding residues as 8 BF16 (lo).
__device__ __forceinline__ void split8(const float (&v)[8], uint4 &hi, uint4 &lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __nv_bfloat162 ph = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        const float2 back = __bfloat1622float2(ph);
        const __nv_bfloat162 pl = __floats2bfloat162_rn(v[2 * i] - back.x, v[2 * i + 1] - back.y);
        h[i] = *reinterpret_cast<const uint32_t *>(&ph);
        l[i] = *reinterpret_cast<const uint32_t *>(&pl);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ uint4 pack8(const float *v) {
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t *>(&p);
    }
    return make_uint4(h[0], h[1], h[2], h[3]);
}

// Column sums over the warp's 32 rows of v[0 .. 31] (columns): lane l returns
// the sum of column l.  Recursive halving, 31 shuffles; destroys v.
__device__ __forceinline__ float column_sum(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int w = 16; w >= 1; w >>= 1) {
#pragma unroll
        for (int i = 0; i < w; i++) {
            const bool up = lane & w;
            const float keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    return v[0];
}

__device__ __forceinline__ uint64_t make_desc_t(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(T_LBO >> 4) << 16) | ((uint64_t)(T_SBO >> 4) << 32) |
           (1ULL << 46);
}

// 32 units [u0, u0 + 32) of sample `row` into a transposed operand.
__device__ __forceinline__ void store_transposed(unsigned char *buf, int row, int u0, const float (&v)[32]) {
    unsigned char *p = buf + (row >> 3) * T_LBO + (row & 7) * 2;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        const int u = u0 + i;
        *reinterpret_cast<__nv_bfloat16 *>(p + (u >> 3) * T_SBO + (u & 7) * 16) = __float2bfloat16_rn(v[i]);
    }
}

// 32 units of sample `row` into a K-major operand (one 16-byte store per 8).
__device__ __forceinline__ void store_rows(unsigned char *buf, int row, int u0, const float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 32; i += 8)
        *reinterpret_cast<uint4 *>(buf + noa_tc::canon_off(row, u0 + i)) = pack8(v + i);
}
__device__ __forceinline__ void store_rows_split(unsigned char *hi, unsigned char *lo, int row, int u0,
                                                 const float (&v)[32]) {
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
            w[j] = v[i + j];
        uint4 h, l;
        split8(w, h, l);
        *reinterpret_cast<uint4 *>(hi + noa_tc::canon_off(row, u0 + i)) = h;
        *reinterpret_cast<uint4 *>(lo + noa_tc::canon_off(row, u0 + i)) = l;
    }
}

// A 128 x 128 BF16 matrix (row-major) into a K-major operand, by asynchronous
// copies of the calling thread's current group.
__device__ __forceinline__ void stage_matrix(unsigned char *buf, const __nv_bfloat16 *W) {
    const uint32_t base = noa_tc::smem_u32(buf);
#pragma unroll
    for (int e = threadIdx.x; e < H * H / 8; e += TILE_THREADS) {
        const int r = e % H, k0 = (e / H) * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + noa_tc::canon_off(r, k0)),
                     "l"(W + r * H + k0)
                     : "memory");
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// One tile of 128 samples through the network (pred), or through the network
// and back (TRAIN: loss and gradient accumulated).  Thread t owns sample
// (t / 32 % 4) 32 + t % 32, its TMEM lane, and the 32 units from 32 (t / 128):
// it computes their activations, writes them as the next product's operands
// and keeps what the way back needs in registers; one thread issues each
// product's MMAs and commits to an mbarrier, every thread waits (bounded).
// The kernel is straight-line code that each warp runs once, so its length
// counts (64 units a thread: 9200 instructions a warp, 4.5 "no instruction"
// stalls an issue, 64 us): each sigmoid is computed once and serves the
// activation and its derivative.
//
// Operands, six buffers of 32 KB:
//   forward   P0 W2 hi, P1 W2 lo, P2 W3 hi, P3 W3 lo, P4 / P5 activations hi / lo
//   backward  P0 W3^T, P1 W2^T (copied from the end of layer 2 on), P2 H_prev^T,
//             P4 dZ, P5 dZ^T:  dZ_prev = dZ W  (acc0),  dW = dZ^T H_prev  (acc1)
// Every buffer is rewritten only after the wait for the product that read it.
template <bool TRAIN>
__global__ void __launch_bounds__(TILE_THREADS, 1) mlp_tile_kernel(const TileArgs a) {
    using namespace noa_tc;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *const P0 = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    unsigned char *const P1 = P0 + MAT_BYTES, *const P2 = P0 + 2 * MAT_BYTES, *const P3 = P0 + 3 * MAT_BYTES,
                        *const P4 = P0 + 4 * MAT_BYTES, *const P5 = P0 + 5 * MAT_BYTES;
    __shared__ float4 sW1[H], sX[H];
    __shared__ float sb1[H], sb2[H], sb3[H], sWo[H], sy[4][H];
    __shared__ float s_sum[3][H];  // dWo, db3, db2
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) unsigned long long mbar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, part = warp >> 2, u0 = part * 32;
    constexpr uint32_t cols = TRAIN ? 256 : 128;

    if (warp == 0)
        tmem_alloc(smem_u32(&tmem_slot), cols);
    if (tid == 0) {
        mbar_init(smem_u32(&mbar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < H) {
        const float *w = a.P + OFF_W1 + tid * IN;
        sW1[tid] = make_float4(w[0], w[1], w[2], w[3]);
        sb1[tid] = a.P[OFF_B1 + tid];
        sb2[tid] = a.P[OFF_B2 + tid];
        sb3[tid] = a.P[OFF_B3 + tid];
        sWo[tid] = a.P[OFF_WO + tid];
    }
    const float bo = a.P[OFF_BO];
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t acc0 = tmem_slot, acc1 = tmem_slot + 128;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t mb = smem_u32(&mbar);
    uint32_t phase = 0;
    bool ok = true;

    // Makes the operands written so far visible and has thread 0 issue.
    auto issue = [&](auto mmas) {
        fence_async_smem();
        fence_before();
        __syncthreads();
        fence_after();
        if (tid == 0) {
            mmas();
            mma_commit(mb);
        }
    };
    // True in every thread when the product is done.
    auto wait = [&]() {
        const bool done = mbar_wait(mb, phase);
        phase ^= 1u;
        fence_after();
        return (bool)__syncthreads_and(done);
    };
    auto forward_mmas = [&](unsigned char *wh, unsigned char *wl) {
        const uint32_t ah = smem_u32(P4), al = smem_u32(P5), bh = smem_u32(wh), bl = smem_u32(wl);
#pragma unroll
        for (int o = 0; o < 8 * 256; o += 256) {  // 16 K-elements = two core matrices
            mma_ss(acc0, make_desc(ah + o), make_desc(bh + o), o > 0);
            mma_ss(acc0, make_desc(al + o), make_desc(bh + o), 1);
            mma_ss(acc0, make_desc(ah + o), make_desc(bl + o), 1);
        }
    };
    auto backward_mmas = [&](unsigned char *wt) {
        const uint32_t d = smem_u32(P4), w = smem_u32(wt), dt = smem_u32(P5), ht = smem_u32(P2);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            mma_ss(acc0, make_desc(d + k * 256), make_desc(w + k * 256), k > 0);
            mma_ss(acc1, make_desc_t(dt + k * 2 * T_LBO), make_desc_t(ht + k * 2 * T_LBO), k > 0);
        }
    };
    // The weight gradient in acc1: row = out unit, 32 in units per thread.
    auto add_dw = [&](float *dW) {
        float v[32];
        tmem_ld32(acc1 + lane_base + (uint32_t)u0, v);
#pragma unroll
        for (int j = 0; j < 32; j += 4)  // 16-byte vector atomics (the weight blocks of G are 16-byte aligned)
            atomicAdd(reinterpret_cast<float4 *>(&dW[row * H + u0 + j]),
                      make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
    };
    // silu(z), and its derivative in d
    auto silu2 = [](float z, float &d) {
        const float g = __fdividef(1.f, 1.f + __expf(-z));
        d = g * (1.f + z * (1.f - g));
        return silu(z);
    };
    auto layer1 = [&](float4 x, int u) {
        const float4 w = sW1[u];
        return fmaf(w.w, x.w, fmaf(w.z, x.z, fmaf(w.y, x.y, fmaf(w.x, x.x, sb1[u]))));
    };

    const int tiles = (a.M + H - 1) / H;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int s = tile * H + row;
        const bool valid = s < a.M;
        const int64_t src = valid ? (a.perm ? (int64_t)a.perm[s] : (int64_t)s) : 0;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid)
            x = make_float4(a.X[src * IN], a.X[src * IN + 1], a.X[src * IN + 2], a.X[src * IN + 3]);
        if (TRAIN || tile == blockIdx.x) {
            stage_matrix(P0, a.Wb);
            stage_matrix(P1, a.Wb + 2 * H * H);
            copies_commit();
            stage_matrix(P2, a.Wb + H * H);
            stage_matrix(P3, a.Wb + 3 * H * H);
            copies_commit();
        }
        if (TRAIN) {
            if (part == 0)
                sX[row] = x;
            if (tid < H)
                s_sum[0][tid] = s_sum[1][tid] = s_sum[2][tid] = 0.f;
        }
        // layer 1 (FP32)
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; j++)
            v[j] = silu(layer1(x, u0 + j));
        store_rows_split(P4, P5, row, u0, v);
        // layer 2
        copies_wait<1>();
        issue([&] { forward_mmas(P0, P1); });
        if (!(ok = wait()))
            break;
        if (TRAIN) {  // the transposed weights of the way back
            stage_matrix(P0, a.Wb + 5 * H * H);
            stage_matrix(P1, a.Wb + 4 * H * H);
            copies_commit();
        }
        float z2[32];
        tmem_ld32(acc0 + lane_base + (uint32_t)u0, z2);
#pragma unroll
        for (int j = 0; j < 32; j++) {
            z2[j] += sb2[u0 + j];
            v[j] = silu(z2[j]);
        }
        store_rows_split(P4, P5, row, u0, v);
        // layer 3
        copies_wait<TRAIN ? 1 : 0>();
        issue([&] { forward_mmas(P2, P3); });
        if (!(ok = wait()))
            break;
        // output layer (FP32); v = h3, d3 = silu'(z3)
        float d3[32], y = 0.f;
        tmem_ld32(acc0 + lane_base + (uint32_t)u0, v);
#pragma unroll
        for (int j = 0; j < 32; j++) {
            v[j] = silu2(v[j] + sb3[u0 + j], d3[j]);
            y = fmaf(sWo[u0 + j], v[j], y);
        }
        sy[part][row] = y;
        __syncthreads();
        y = bo + ((sy[0][row] + sy[1][row]) + (sy[2][row] + sy[3][row]));
        if (!TRAIN) {
            if (part == 0 && valid)
                a.pred[s] = y;
            fence_before();  // this tile's TMEM reads before the next tile's products
            __syncthreads();
            fence_after();
            continue;
        }
        // loss and its gradient
        const float d = valid ? y - a.T[src] : 0.f;
        const float dp = 2.f * d * a.inv_batch;
        if (part == 0) {
            float l = d * d * a.inv_batch, b = dp;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                l += __shfl_xor_sync(0xffffffffu, l, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
            }
            if (lane == 0) {
                atomicAdd(a.loss, l);
                atomicAdd(&a.G[OFF_BO], b);
            }
        }
        // dZ3, H2^T; dWo, db3; z2 becomes silu'(z2)
#pragma unroll
        for (int j = 0; j < 32; j++) {
            v[j] *= dp;
            d3[j] *= dp * sWo[u0 + j];
        }
        atomicAdd(&s_sum[0][u0 + lane], column_sum(v));
        store_rows(P4, row, u0, d3);
        store_transposed(P5, row, u0, d3);
        atomicAdd(&s_sum[1][u0 + lane], column_sum(d3));
#pragma unroll
        for (int j = 0; j < 32; j++)
            v[j] = silu2(z2[j], z2[j]);
        store_transposed(P2, row, u0, v);
        // dW3 = dZ3^T H2, dZ2 = (dZ3 W3) silu'(Z2)
        copies_wait<0>();
        issue([&] { backward_mmas(P0); });
        if (!(ok = wait()))
            break;
        add_dw(a.G + OFF_W3);
        tmem_ld32(acc0 + lane_base + (uint32_t)u0, v);
#pragma unroll
        for (int j = 0; j < 32; j++)
            v[j] *= z2[j];
        store_rows(P4, row, u0, v);
        store_transposed(P5, row, u0, v);
        atomicAdd(&s_sum[2][u0 + lane], column_sum(v));
#pragma unroll
        for (int j = 0; j < 32; j++)
            v[j] = silu2(layer1(x, u0 + j), z2[j]);  // z2: silu'(z1)
        store_transposed(P2, row, u0, v);
        // dW2 = dZ2^T H1, dZ1 = (dZ2 W2) silu'(Z1)
        issue([&] { backward_mmas(P1); });
        if (!(ok = wait()))
            break;
        add_dw(a.G + OFF_W2);
        // layer 1: dZ1 in FP32 through shared memory (rows of 129 words over the
        // staged weights), then a thread per unit and quarter of the samples
        float *D1 = reinterpret_cast<float *>(P0);
        tmem_ld32(acc0 + lane_base + (uint32_t)u0, v);
#pragma unroll
        for (int j = 0; j < 32; j++)
            D1[row * (H + 1) + u0 + j] = v[j] * z2[j];
        fence_before();
        __syncthreads();
        fence_after();
        {
            const int j = tid & (H - 1), first = (tid >> 7) * 32;
            float gb = 0.f, gw[IN] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int i = first; i < first + 32; i++) {
                const float g = D1[i * (H + 1) + j];
                const float4 xi = sX[i];
                gb += g;
                gw[0] = fmaf(g, xi.x, gw[0]);
                gw[1] = fmaf(g, xi.y, gw[1]);
                gw[2] = fmaf(g, xi.z, gw[2]);
                gw[3] = fmaf(g, xi.w, gw[3]);
            }
#pragma unroll
            for (int c = 0; c < IN; c++)
                atomicAdd(&a.G[OFF_W1 + j * IN + c], gw[c]);
            atomicAdd(&a.G[OFF_B1 + j], gb);
        }
        if (tid < H) {
            atomicAdd(&a.G[OFF_WO + tid], s_sum[0][tid]);
            atomicAdd(&a.G[OFF_B3 + tid], s_sum[1][tid]);
            atomicAdd(&a.G[OFF_B2 + tid], s_sum[2][tid]);
        }
        __syncthreads();  // the next tile stages over D1 and clears the sums
    }
    if (!ok) {
        if (tid == 0)
            atomicMax(a.status, (unsigned int)NOA_DCS_ERROR_TIMEOUT);
        mbar_wait(mb, phase ^ 1u);  // one more bounded wait before the TMEM it writes is freed
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 0)
        tmem_dealloc(acc0, cols);
}

// The BF16 forms of W2, W3 that the products read, six 128 x 128 matrices: W2
// hi, W3 hi, W2 lo, W3 lo, and W2 hi, W3 hi transposed (the way back).
//
// UPDATE_CTAS CTAs of 1024 threads cover the parameters, one each: the first
// 32 CTAs a 32 x 32 block of W2 or W3 each (its transposed half through shared
// memory, so that both are written in rows), the others the rest.  f(i) gives
// parameter i's new value.
constexpr int UPDATE_CTAS = 32 + 2, UPDATE_THREADS = 1024;
template <typename F>
__device__ __forceinline__ void update_parameters(__nv_bfloat16 *Wb, F f) {
    __shared__ __nv_bfloat16 t[32][33];
    const int c = threadIdx.x & 31, r = threadIdx.x >> 5;
    // W1 b1 | b2 | b3 Wo bo
    constexpr int n1 = OFF_W2, n2 = n1 + H, n3 = n2 + NPARAM - OFF_B3;
    static_assert((UPDATE_CTAS - 32) * UPDATE_THREADS >= n3, "every parameter has a thread");
    const bool block = blockIdx.x < 32;
    const int layer = blockIdx.x >> 4, row = (blockIdx.x >> 2 & 3) * 32, col = (blockIdx.x & 3) * 32;
    const int w = (row + r) * H + col + c;
    const int k = ((int)blockIdx.x - 32) * UPDATE_THREADS + threadIdx.x;
    if (!block && k >= n3)
        return;
    const float p = f(block ? (layer ? OFF_W3 : OFF_W2) + w
                            : (k < n1 ? k : (k < n2 ? OFF_B2 + k - n1 : OFF_B3 + k - n2)));
    if (block) {
        const __nv_bfloat16 hi = __float2bfloat16_rn(p);
        Wb[layer * H * H + w] = hi;
        Wb[(2 + layer) * H * H + w] = __float2bfloat16_rn(p - __bfloat162float(hi));
        t[r][c] = hi;
        __syncthreads();
        Wb[(4 + layer) * H * H + (col + r) * H + row + c] = t[c][r];
    }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters; refreshes the BF16
// weights, hands the step's loss out and leaves gradient and loss zero for
// the next step.
__global__ void __launch_bounds__(UPDATE_THREADS) mlp_adam_kernel(float *P, float *G, float *Mm, float *V, __nv_bfloat16 *Wb,
                                                       float lr, float b1, float b2, float eps, float c1, float c2,
                                                       float *loss, float *loss_out) {
    update_parameters(Wb, [&](int i) {
        const float g = G[i];
        G[i] = 0.f;
        const float m = b1 * Mm[i] + (1.f - b1) * g;
        const float v = b2 * V[i] + (1.f - b2) * g * g;
        Mm[i] = m;
        V[i] = v;
        const float p = P[i] - lr * (m * c1) / (sqrtf(v * c2) + eps);
        P[i] = p;
        return p;
    });
    if (blockIdx.x == 32 && threadIdx.x == 0) {
        if (loss_out)
            *loss_out = *loss;
        *loss = 0.f;
    }
}

__global__ void __launch_bounds__(UPDATE_THREADS) mlp_round_weights_kernel(const float *P, __nv_bfloat16 *Wb) {
    update_parameters(Wb, [&](int i) { return P[i]; });
}

// Training data: raw features and the residual target from the FP64 plain
// kernels (dcs_fp64.cuh).  state: 1 = open pair with DCS > 0 (a training
// sample), 0 = closed by the kinematic bounds, 2 = open by the bounds but with
// DCS = 0 (every screening term clamped) or no finite baseline -- cells that
// hold such pairs must not be answered by the network.
template <int PROC>
__global__ void mlp_prepare_kernel(const double *K, const double *q, const uint8_t *elem, int64_t n,
                                   const noa_dcs_consts *consts, const float *logA, float *Xraw, float *R,
                                   uint8_t *valid) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const noa_dcs_consts &c = consts[elem[i]];
        double base;
        const bool open = baseline<PROC>(K[i], q[i], c, base);
        bool ok = open;
        double d = 0.;
        if (ok) {
            d = PROC == NOA_DCS_PAIR_PRODUCTION ? noa_dcs::pprod_fp64(K[i], q[i], c) : noa_dcs::photo_fp64(K[i], q[i], c);
            ok = d > 0. && isfinite(base);
        }
        const double nu = q[i] / (K[i] + c.mass);
        Xraw[i * IN + 0] = (float)log(K[i]);
        Xraw[i * IN + 1] = (float)log(nu);
        Xraw[i * IN + 2] = (float)c.Zd * 0.01f;
        Xraw[i * IN + 3] = logA[elem[i]];
        R[i] = ok ? (float)(log(d) - base) : 0.f;
        valid[i] = ok ? 1 : (open ? 2 : 0);
    }
}

} // namespace

struct noa_dcs_mlp {
    int process = 0;
    int batch = 0;
    float *P = nullptr, *G = nullptr, *Mm = nullptr, *V = nullptr;
    __nv_bfloat16 *Wb = nullptr;
    float *loss = nullptr;
    unsigned int *status = nullptr;  // device word, see take_status
    int64_t step = 0;
    float norm[2 * IN + 2] = {};
};

namespace {

thread_local char g_merr[256] = "";

int mfail(int st, const char *msg, cudaError_t e = cudaSuccess) {
    if (e != cudaSuccess)
        snprintf(g_merr, sizeof g_merr, "%s: %s", msg, cudaGetErrorString(e));
    else
        snprintf(g_merr, sizeof g_merr, "%s", msg);
    return st;
}

// Raises the tile kernels' dynamic shared-memory limits once per device
// (called when a model is created).
cudaError_t set_tile_smem() {
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return e;
    if (dev >= 0 && dev < 64 && done[dev].load())
        return cudaSuccess;
    e = cudaFuncSetAttribute(mlp_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM);
    if (e == cudaSuccess && dev >= 0 && dev < 64)
        done[dev].store(true);
    return e;
}

// Status word of the tensor-core kernels: NOA_DCS_ERROR_TIMEOUT after an
// expired mbarrier wait.  Read (and cleared) after the work of a call;
// synchronises the stream.
int take_status(noa_dcs_mlp *m, cudaStream_t s);

int sm_count() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// Prediction (pred) of M rows of X, or, with targets T, their loss and
// gradient added to m->loss and m->G; rows perm[0 .. M) of X and T if given.
cudaError_t run_tiles(noa_dcs_mlp *m, const float *X, const float *T, const int32_t *perm, int M, float *pred,
                      cudaStream_t s) {
    TileArgs a{};
    a.X = X;
    a.T = T;
    a.perm = perm;
    a.P = m->P;
    a.Wb = m->Wb;
    a.G = m->G;
    a.loss = m->loss;
    a.pred = pred;
    a.status = m->status;
    a.inv_batch = 1.f / (float)M;
    a.M = M;
    const int tiles = (M + H - 1) / H, sms = sm_count();
    const int grid = tiles < sms ? tiles : sms;
    if (T)
        mlp_tile_kernel<true><<<grid, TILE_THREADS, TILE_SMEM, s>>>(a);
    else
        mlp_tile_kernel<false><<<grid, TILE_THREADS, TILE_SMEM, s>>>(a);
    return cudaGetLastError();
}

cudaError_t clear_gradient(noa_dcs_mlp *m, cudaStream_t s) {
    const cudaError_t e = cudaMemsetAsync(m->G, 0, sizeof(float) * NPARAM, s);
    return e == cudaSuccess ? cudaMemsetAsync(m->loss, 0, sizeof(float), s) : e;
}

// Every buffer must be device (or managed) memory of the current device before
// it reaches a kernel; nullptr passes (optional arguments are checked by the
// callers).
bool device_ok(std::initializer_list<const void *> ptrs) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return false;
    for (const void *p : ptrs) {
        if (!p)
            continue;
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (!(a.type == cudaMemoryTypeManaged || (a.type == cudaMemoryTypeDevice && a.device == dev)))
            return false;
    }
    return true;
}

int take_status(noa_dcs_mlp *m, cudaStream_t s) {
    unsigned int st = 0;
    cudaError_t e = cudaMemcpyAsync(&st, m->status, sizeof st, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "status read", e);
    if (st) {
        cudaMemsetAsync(m->status, 0, sizeof st, s);
        return mfail((int)st, "a tensor-core wait expired (mbarrier); the results of this call are invalid");
    }
    return NOA_DCS_SUCCESS;
}

} // namespace

extern "C" {

int noa_dcs_mlp_create(noa_dcs_mlp **out, int process, int batch) {
    g_merr[0] = '\0';
    if (!out)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "NULL model pointer");
    *out = nullptr;
    if (process != NOA_DCS_PAIR_PRODUCTION && process != NOA_DCS_PHOTONUCLEAR)
        return mfail(NOA_DCS_ERROR_NOT_SUPPORTED, "the surrogate covers pair production and photonuclear");
    if (batch < 128 || batch > (1 << 20) || batch % 128)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "batch must be a multiple of 128 in [128, 2^20]");
    cudaError_t e = set_tile_smem();
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "cudaFuncSetAttribute", e);
    noa_dcs_mlp *m = new (std::nothrow) noa_dcs_mlp();
    if (!m)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "out of host memory");
    m->process = process;
    m->batch = batch;
    e = cudaMalloc((void **)&m->P, sizeof(float) * NPARAM_PAD * 4);
    if (e == cudaSuccess)
        e = cudaMalloc((void **)&m->Wb, sizeof(__nv_bfloat16) * 6 * H * H);
    if (e == cudaSuccess)
        e = cudaMalloc((void **)&m->loss, 2 * sizeof(float));
    if (e != cudaSuccess) {
        cudaFree(m->P);
        cudaFree(m->Wb);
        cudaFree(m->loss);
        delete m;
        return mfail(NOA_DCS_ERROR_CUDA, "model allocation", e);
    }
    m->G = m->P + NPARAM_PAD;  // each block 16-byte aligned (vector atomics on G)
    m->Mm = m->G + NPARAM_PAD;
    m->V = m->Mm + NPARAM_PAD;
    m->status = reinterpret_cast<unsigned int *>(m->loss + 1);
    cudaMemset(m->P, 0, sizeof(float) * NPARAM_PAD * 4);
    cudaMemset(m->status, 0, sizeof(unsigned int));
    cudaMemset(m->Wb, 0, sizeof(__nv_bfloat16) * 6 * H * H);
    *out = m;
    return NOA_DCS_SUCCESS;
}

int noa_dcs_mlp_set_params(noa_dcs_mlp *m, const float *params, const float *adam_m, const float *adam_v,
                           int64_t step, const float *norm) {
    if (!m || !params || !norm)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "NULL argument");
    cudaError_t e = cudaMemcpy(m->P, params, sizeof(float) * NPARAM, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = adam_m ? cudaMemcpy(m->Mm, adam_m, sizeof(float) * NPARAM, cudaMemcpyHostToDevice)
                   : cudaMemset(m->Mm, 0, sizeof(float) * NPARAM);
    if (e == cudaSuccess)
        e = adam_v ? cudaMemcpy(m->V, adam_v, sizeof(float) * NPARAM, cudaMemcpyHostToDevice)
                   : cudaMemset(m->V, 0, sizeof(float) * NPARAM);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "cudaMemcpy(params)", e);
    mlp_round_weights_kernel<<<UPDATE_CTAS, UPDATE_THREADS>>>(m->P, m->Wb);
    if ((e = cudaDeviceSynchronize()) != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "round weights", e);
    m->step = step;
    std::memcpy(m->norm, norm, sizeof m->norm);
    return NOA_DCS_SUCCESS;
}

int noa_dcs_mlp_get_params(noa_dcs_mlp *m, float *params, float *adam_m, float *adam_v, int64_t *step) {
    if (!m || !params)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "NULL argument");
    cudaError_t e = cudaMemcpy(params, m->P, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && adam_m)
        e = cudaMemcpy(adam_m, m->Mm, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && adam_v)
        e = cudaMemcpy(adam_v, m->V, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "cudaMemcpy(params)", e);
    if (step)
        *step = m->step;
    return NOA_DCS_SUCCESS;
}

int noa_dcs_mlp_prepare(int process, const double *K, const double *q, const uint8_t *elem, int64_t n,
                        const noa_dcs_element *elements, int n_elements, double mass, float *Xraw, float *R,
                        uint8_t *valid, void *stream) {
    g_merr[0] = '\0';
    if (process != NOA_DCS_PAIR_PRODUCTION && process != NOA_DCS_PHOTONUCLEAR)
        return mfail(NOA_DCS_ERROR_NOT_SUPPORTED, "the surrogate covers pair production and photonuclear");
    if (n < 0 || n_elements < 1 || n_elements > 16 || !elements)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "bad sizes");
    if (n == 0)
        return NOA_DCS_SUCCESS;
    if (!K || !q || !elem || !Xraw || !R || !valid || !device_ok({K, q, elem, Xraw, R, valid}))
        return mfail(NOA_DCS_ERROR_NOT_DEVICE_MEMORY, "K, q, elem, Xraw, R and valid must be device memory");
    noa_dcs_consts hc[16];
    float hlogA[16];
    for (int i = 0; i < n_elements; i++) {
        noa_dcs_fill_consts(&hc[i], elements[i].A, elements[i].I, elements[i].Z, mass);
        hlogA[i] = (float)std::log(elements[i].A);
    }
    // The element table (up to 16 constant sets) is staged through a small
    // device buffer that lives until this call's work is done (synchronised
    // below); data preparation is off the evaluation path.
    noa_dcs_consts *dc = nullptr;
    float *dl = nullptr;
    cudaError_t e = cudaMalloc((void **)&dc, sizeof hc + sizeof hlogA);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "cudaMalloc(element table)", e);
    dl = reinterpret_cast<float *>(dc + 16);
    cudaStream_t s = (cudaStream_t)stream;
    e = cudaMemcpyAsync(dc, hc, sizeof hc, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dl, hlogA, sizeof hlogA, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        const int64_t blocks = (n + 255) / 256;
        const int grid = (int)(blocks < 152 * 16 ? blocks : 152 * 16);
        if (process == NOA_DCS_PAIR_PRODUCTION)
            mlp_prepare_kernel<NOA_DCS_PAIR_PRODUCTION><<<grid, 256, 0, s>>>(K, q, elem, n, dc, dl, Xraw, R, valid);
        else
            mlp_prepare_kernel<NOA_DCS_PHOTONUCLEAR><<<grid, 256, 0, s>>>(K, q, elem, n, dc, dl, Xraw, R, valid);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    cudaFree(dc);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "prepare", e);
    return NOA_DCS_SUCCESS;
}

int noa_dcs_mlp_train(noa_dcs_mlp *m, const float *X, const float *T, int64_t n, const int32_t *perm,
                      int64_t n_steps, float lr, float lr_final, float *losses, void *stream) {
    g_merr[0] = '\0';
    if (!m || !X || !T || !perm || n < m->batch || n_steps < 0)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "bad training arguments (n must be at least one batch)");
    if (!device_ok({X, T, perm, losses}))
        return mfail(NOA_DCS_ERROR_NOT_DEVICE_MEMORY, "X, T, perm and losses must be device memory");
    cudaStream_t s = (cudaStream_t)stream;
    const int B = m->batch;
    const int64_t batches = n / B;
    cudaError_t e = clear_gradient(m, s);
    for (int64_t i = 0; i < n_steps && e == cudaSuccess; i++) {
        const int64_t b = (m->step) % batches;
        if ((e = run_tiles(m, X, T, perm + b * B, B, nullptr, s)) != cudaSuccess)
            break;
        // cosine decay from lr to lr_final over the n_steps of this call
        const double frac = n_steps > 1 ? (double)i / (double)(n_steps - 1) : 0.;
        const float lr_i = (float)(lr_final + 0.5 * (lr - lr_final) * (1. + std::cos(M_PI * frac)));
        m->step++;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f / (1.f - std::pow(b1, (float)m->step));
        const float c2 = 1.f / (1.f - std::pow(b2, (float)m->step));
        mlp_adam_kernel<<<UPDATE_CTAS, UPDATE_THREADS, 0, s>>>(m->P, m->G, m->Mm, m->V, m->Wb, lr_i, b1, b2, 1e-8f,
                                                             c1, c2, m->loss, losses ? losses + i : nullptr);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "training step", e);
    return take_status(m, s);
}

int noa_dcs_mlp_predict(noa_dcs_mlp *m, const float *X, float *out, int64_t n, void *stream) {
    g_merr[0] = '\0';
    if (!m || (n > 0 && (!X || !out)) || n < 0)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "bad arguments");
    if (n > 0 && !device_ok({X, out}))
        return mfail(NOA_DCS_ERROR_NOT_DEVICE_MEMORY, "X and out must be device memory");
    cudaStream_t s = (cudaStream_t)stream;
    constexpr int64_t most = (int64_t)1 << 24;  // rows of one launch
    for (int64_t off = 0; off < n; off += most) {
        const int M = (int)(n - off < most ? n - off : most);
        const cudaError_t e = run_tiles(m, X + off * IN, nullptr, nullptr, M, out + off, s);
        if (e != cudaSuccess)
            return mfail(NOA_DCS_ERROR_CUDA, "forward", e);
    }
    return n > 0 ? take_status(m, s) : NOA_DCS_SUCCESS;
}

int noa_dcs_mlp_gradient(noa_dcs_mlp *m, const float *X, const float *T, int n, float *grad, float *loss,
                         void *stream) {
    g_merr[0] = '\0';
    if (!m || !X || !T || !grad || n < 1 || n > m->batch)
        return mfail(NOA_DCS_ERROR_INVALID_VALUE, "bad arguments (1 <= n <= batch)");
    if (!device_ok({X, T, grad, loss}))
        return mfail(NOA_DCS_ERROR_NOT_DEVICE_MEMORY, "X, T, grad and loss must be device memory");
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = clear_gradient(m, s);
    if (e == cudaSuccess)
        e = run_tiles(m, X, T, nullptr, n, nullptr, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(grad, m->G, sizeof(float) * NPARAM, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess && loss)
        e = cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess)
        return mfail(NOA_DCS_ERROR_CUDA, "gradient", e);
    return take_status(m, s);
}

int noa_dcs_mlp_destroy(noa_dcs_mlp *m) {
    if (!m)
        return NOA_DCS_SUCCESS;
    cudaFree(m->P);
    cudaFree(m->Wb);
    cudaFree(m->loss);
    delete m;
    return NOA_DCS_SUCCESS;
}

const char *noa_dcs_mlp_last_error(void) { return g_merr; }

// Internal accessor for the inference translation unit (mlp_infer.cu).
int noa_dcs_mlp_handles(noa_dcs_mlp *m, int *process, const float **P, const void **Wb, const float **norm) {
    if (!m)
        return 1;
    *process = m->process;
    *P = m->P;
    *Wb = m->Wb;
    *norm = m->norm;
    return 0;
}

} // extern "C"
