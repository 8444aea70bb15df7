/*
 * FP64-accurate elementary functions that issue few FP64 instructions.
 *
 * On GB300 the FP64 pipe retires 2 lanes per clock per SM: one FP64 warp
 * instruction occupies it for 16 clocks, while the SM issues 4 warp
 * instructions per clock to its integer (ALU, 64 lanes) and FP32 (128 lanes)
 * pipes.  A DCS kernel built on FP64 arithmetic is therefore bound by its
 * FP64 instruction count with issue ~80% idle (ncu: FP64 pipe 86%, issue
 * 12%), and replacing one FP64 instruction by up to ~30 integer or FP32
 * instructions still shortens it.  The functions here keep double accuracy
 * (0.5 - 0.9 ulp; tests compare them with CUDA's functions and numpy) and do
 * their work in exact 64-bit integer arithmetic (range reduction, products
 * with short table constants, fixed-point sums rounded once to double) and
 * in float-float arithmetic (the small correction terms, which need 2^-47
 * relative).  What they spend is ALU issue (64 lanes: shifts, selects, 64-bit
 * adds), so values cross between float and integer through the FMA pipe
 * (integers carried in the low bits of a float, products by powers of two
 * instead of shifts) or as the two 32-bit words of a fixed-point number,
 * never by normalising.  Four processes x 3e7 pairs: 42.2 ms with the same
 * methods at 1 / 2 / 0 FP64 instructions and normalised conversions (about
 * twice the ALU instructions), 35.3 ms with these in the same bodies:
 *
 *   lean_log   0 FP64 ops.  Tang's table method (P. T. P. Tang, ACM TOMS
 *              16(4), 1990): x = 2^e m, c_t ~ 1/m with 11 fractional bits from
 *              the top 9 mantissa bits; r = m c_t - 1 exact in 64-bit integers;
 *              log x = e ln2 - log c_t + r + (log1p(r) - r), summed in 64-bit
 *              fixed point at a scale that follows |e| and rounded once.
 *              Within 2^-9 of 1 c = 1 and the scale follows r: full
 *              relative accuracy near 1.
 *   lean_exp   0 FP64 ops.  Tang's table method (ACM TOMS 15(2), 1989): x as a
 *              64-bit fixed-point number, k = round(x 128 / ln2),
 *              r = x - k ln2 / 128 modulo 2^64, expm1(r) - r in float-float,
 *              2^k' T_j (1 + expm1 r) by integer products, rounded once.
 *   lean_rcp   0 FP64 ops.  MUFU seed y0 as an integer, the exact residual
 *              1 - m y0 by one 64-bit integer product, y0 (1 + e + e^2) in
 *              fixed point, rounded once.
 *   lean_div   1 FP64 op: a * lean_rcp(b).
 *   lean_sqrt  6 FP64 ops.  MUFU rsqrt, then two Newton steps on s = x y.
 *
 * Arguments outside the fast range (zero, negative, subnormal, |x| > 700
 * for exp, |b| >= 2^1022 for rcp, values outside float range for sqrt,
 * inf, NaN) take CUDA's IEEE function, so special values behave exactly as
 * in IEEE arithmetic.  The double <-> float and int -> double conversions go
 * through the integer pipe (fpconv.cuh), because the hardware conversions
 * would occupy the FP64 pipe too.
 */
#pragma once

#include "fpconv.cuh"
#include "lean64_tables.h"

#include <cstring>

#include <cuda_runtime.h>

namespace lean64 {

#ifndef LEAN64_FN
#define LEAN64_FN __device__ __forceinline__
#endif

LEAN64_FN float rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    // host builds: a stand-in seed 1 - 3 ulp off the rounded 1/x, as far off
    // as the MUFU approximation may be, so that host checks cover that error
    float r = 1.f / x;
    unsigned u;
    memcpy(&u, &r, 4);
    u ^= 3u;
    memcpy(&r, &u, 4);
    return r;
#endif
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x >= 0 finite double compared with a positive constant through the bit
// pattern (integer pipe); NaN compares as larger than every constant.
__device__ __forceinline__ bool bits_ge(double x, double c) {
    return __double_as_longlong(x) >= __double_as_longlong(c);
}

// ------------------------------------------------------------ lean_log / lean_exp
// Host builds of lean_log / lean_exp / lean_rcp (for checking them on a CPU)
// define LEAN64_FN as __host__ __device__ and LEAN64_HOST_TABLES before
// including this header; the product builds them for the device only.

#if defined(LEAN64_HOST_TABLES) && !defined(__CUDA_ARCH__)
static const longlong2 lean64_log_tab_host[1 << LEAN64_LOG_BITS] = LEAN64_LOG_TAB_DATA;
static const long long lean64_exp_t_host[LEAN64_EXP_N] = LEAN64_EXP_TAB_DATA;
#endif

namespace detail {

#if defined(__CUDA_ARCH__) || !defined(LEAN64_HOST_TABLES)
__device__ __forceinline__ long long d2ll(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double ll2d(long long b) { return __longlong_as_double(b); }
__device__ __forceinline__ unsigned f2u(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float u2f(unsigned b) { return __uint_as_float(b); }
__device__ __forceinline__ int clz64(unsigned long long x) { return __clzll((long long)x); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ int clz32(unsigned x) { return __clz((int)x); }
__device__ __forceinline__ float i2f(int i) { return __int2float_rn(i); }
__device__ __forceinline__ unsigned mulhi_s(int a, int b) { return (unsigned)__mulhi(a, b); }
__device__ __forceinline__ unsigned long long mulhi_u64(unsigned long long a, unsigned long long b) {
    return __umul64hi(a, b);
}
__device__ __forceinline__ long long mulhi_s64(long long a, long long b) { return __mul64hi(a, b); }
__device__ __forceinline__ longlong2 log_entry(int t) { return __ldg(&lean64_log_tab[t]); }
__device__ __forceinline__ long long exp_entry(int j) { return __ldg(&lean64_exp_t[j]); }
#elif defined(LEAN64_HOST_TABLES)
inline long long d2ll(double x) { long long b; memcpy(&b, &x, 8); return b; }
inline double ll2d(long long b) { double x; memcpy(&x, &b, 8); return x; }
inline unsigned f2u(float x) { unsigned b; memcpy(&b, &x, 4); return b; }
inline float u2f(unsigned b) { float x; memcpy(&x, &b, 4); return x; }
inline int clz64(unsigned long long x) { return __builtin_clzll(x); }
inline float fadd(float a, float b) { return a + b; }  // host code is built with -ffp-contract=off
inline float fmul(float a, float b) { return a * b; }
inline int clz32(unsigned x) { return __builtin_clz(x); }
inline float i2f(int i) { return (float)i; }
inline unsigned mulhi_s(int a, int b) { return (unsigned)(((long long)a * b) >> 32); }
inline unsigned long long mulhi_u64(unsigned long long a, unsigned long long b) {
    return (unsigned long long)(((unsigned __int128)a * b) >> 64);
}
inline long long mulhi_s64(long long a, long long b) { return (long long)(((__int128)a * b) >> 64); }
inline longlong2 log_entry(int t) { return lean64_log_tab_host[t]; }
inline long long exp_entry(int j) { return lean64_exp_t_host[j]; }
#endif

// f 2^F as a signed 64-bit integer, truncated toward zero; 0 for zero and
// float subnormals.  Callers keep |f| 2^F below 2^55 (a left shift <= 31).
LEAN64_FN long long fix_from_float(float f, int F) {
    const unsigned u = f2u(f);
    const unsigned ef = (u >> 23) & 0xFFu;
    // the significand (implicit bit set) at bits 40..63: the float's
    // exponent and sign bits fall off the top of the word
    const unsigned long long m = (unsigned long long)(u | 0x800000u) << 40;
    const int t = 190 - (int)ef - F;  // bit 0 of the significand weighs 2^(ef - 150); t >= 9
    const unsigned long long v = (ef != 0u && t < 64) ? (m >> t) : 0ull;
    return (u >> 31) ? -(long long)v : (long long)v;
}

// S 2^-F as a double, rounded to nearest even; S != 0, 1 <= 1086 - F - clz.
LEAN64_FN double fix_to_double(long long S, int F) {
    const unsigned long long sign = (unsigned long long)S & 0x8000000000000000ull;
    const unsigned long long U = S < 0 ? 0ull - (unsigned long long)S : (unsigned long long)S;
    const int lz = clz64(U);
    const unsigned long long N = U << lz;  // leading bit at 63
    unsigned long long m = N >> 11;        // 53 bits, leading bit at 52
    const unsigned long long rest = N & 0x7FFull;
    m += (rest > 0x400ull || (rest == 0x400ull && (m & 1ull))) ? 1ull : 0ull;
    // biased exponent 1086 - lz - F; the leading bit of m adds the last 1
    // (and a carry out of rounding moves to the next binade by itself)
    return ll2d((long long)(sign | (((unsigned long long)(1085 - lz - F) << 52) + m)));
}

// Z 2^-F as a double, rounded half up in the last place, for |Z| >= 2^32: the
// leading bit is then in the high word (one 32-bit count).  Z is a value cut
// downwards; the one's complement of a negative Z is its magnitude cut
// downwards, so that the last rounding is that of the uncut value.
LEAN64_FN double fix_wide_to_double(long long Z, int F) {
    const unsigned long long U = (unsigned long long)(Z ^ (Z >> 63));
    const int lz = clz32((unsigned)(U >> 32)) - 1;  // the caller keeps |Z| < 2^63
    const unsigned long long m = ((U << lz) + 0x200ull) >> 10;  // leading bit at 52
    return ll2d((long long)((((unsigned long long)(1084 - lz - F) << 52) + m) |
                            ((unsigned long long)Z & 0x8000000000000000ull)));
}

// The pair dh + dl as an integer in units of 2^-(S + 22), in two parts that
// float adds round: i1 = round(d 2^S), i2 = round((d 2^S - i1) 2^22).  Returns
// their float carriers, whose offsets the caller's constants take off:
// `magic` (1.5 2^23 for |d| 2^S < 2^22, 2^24 - 1 for -2^23 < d 2^S <= 0) and
// 1.5 2^23.
LEAN64_FN void fix_parts(float dh, float dl, float scale, float magic, unsigned &b1, unsigned &b2) {
    const float t1 = fmaf(fadd(dh, dl), scale, magic);
    const float g = fmaf(dl, scale, fmaf(dh, scale, -fadd(t1, -magic)));
    b1 = f2u(t1);
    b2 = f2u(fmaf(g, 4194304.f, 12582912.f));
}

// d = log1p(r) - r as dh + dl, r = R 2^-64, |r| < 2^-9.
LEAN64_FN void log_tail(long long R, float &dh, float &dl) {
    // r = rh + rl: the high word rounded and the signed low word, renormalised
    const float rw = fmul(i2f((int)((R + 0x80000000ll) >> 32)), 0x1p-32f);
    const float rv = fmul(i2f((int)(unsigned)R), 0x1p-64f);
    const float rh = fadd(rw, rv);
    const float rl = fadd(rv, -fadd(rh, -rw));
    // d = -r^2/2 + r^3 w,  w = 1/3 - r/4 + r^2 (1/5 - r/6 + r^2/7); the last
    // term is below 2^-63 but in the window around 1
    const float sh = fmul(rh, rh);
    const float sl = fmaf(fmul(2.f, rh), rl, fmaf(rh, rh, -sh));
    const float zt = fmul(sh, fmaf(rh, fmaf(rh, 1.f / 7.f, -1.f / 6.f), 0.2f));
    const float qa = fmul(-0.25f, rh);
    const float zh = fadd(qa, zt);
    const float zl = fmaf(-0.25f, rl, fadd(zt, -fadd(zh, -qa)));
    const float wh = fadd(LEAN64_THIRD_H, zh);
    const float wl = fadd(fadd(zh, -fadd(wh, -LEAN64_THIRD_H)), fadd(zl, LEAN64_THIRD_L));
    const float ch = fmul(sh, rh);
    const float cl = fmaf(sh, rl, fmaf(sl, rh, fmaf(sh, rh, -ch)));
    const float uh = fmul(ch, wh);
    const float ul = fmaf(ch, wl, fmaf(cl, wh, fmaf(ch, wh, -uh)));
    const float hs = fmul(-0.5f, sh);
    dh = fadd(hs, uh);
    dl = fadd(fadd(uh, -fadd(dh, -hs)), fmaf(-0.5f, sl, ul));
}

// log of the table bin's m (see lean_log) from R and the bin's L, in units of 2^-64.
LEAN64_FN long long log_bin(long long R, long long L) {
    float dh, dl;
    log_tail(R, dh, dl);
    unsigned b1, b2;
    fix_parts(dh, dl, 0x1p42f, 16777215.f, b1, b2);  // -2^-19.9 < d <= 0
    return R + (long long)((unsigned long long)L + (unsigned long long)b1 * 0x400000ull + b2);
}

// exp: k ln2 / 128 in units of 2^-63, modulo 2^64 (unsigned, as its first part and
// the sum wrap).
LEAN64_FN unsigned long long k_ln2n(int k) {
    return (unsigned long long)((long long)k * LEAN64_K_M) +
           ((unsigned long long)((unsigned)k * (unsigned)LEAN64_K_H) << 32) +
           (unsigned long long)(long long)(int)mulhi_s(k, LEAN64_K_L);
}

// exp: T_j (1 + expm1 r) in units of 2^-61, in [2^61, 2^62), for k = 128 k' + j
// and r = R 2^-63, |r| < 2^-8.4; q = k' or, where T_0 (1 + expm1 r) < 1, k' - 1.
LEAN64_FN unsigned long long exp_bin(int k, long long r, int &q) {
    // r = rh + rl: the high word rounded and the signed low word
    const float rh = fmul(i2f((int)((r + 0x80000000ll) >> 32)), 0x1p-31f);
    const float rl = fmul(i2f((int)(unsigned)r), 0x1p-63f);
    // d = r^2 (1/2 + r w),  w = 1/6 + r (1/24 + r (1/120 + r/720))
    const float sh = fmul(rh, rh);
    const float sl = fmaf(fmul(2.f, rh), rl, fmaf(rh, rh, -sh));
    const float g = fmul(rh, fmaf(rh, fmaf(rh, 1.f / 720.f, 1.f / 120.f), 1.f / 24.f));
    const float wh = fadd(LEAN64_SIXTH_H, g);
    const float wl = fadd(fadd(g, -fadd(wh, -LEAN64_SIXTH_H)), LEAN64_SIXTH_L);
    const float vh = fmul(rh, wh);
    const float vl = fmaf(rh, wl, fmaf(rl, wh, fmaf(rh, wh, -vh)));
    const float qh = fadd(0.5f, vh);
    const float ql = fadd(fadd(vh, -fadd(qh, -0.5f)), vl);
    const float dh = fmul(sh, qh);
    const float dl = fmaf(sh, ql, fmaf(sl, qh, fmaf(sh, qh, -dh)));
    // p = r + d in units of 2^-63
    unsigned b1, b2;
    fix_parts(dh, dl, 0x1p39f, 12582912.f, b1, b2);
    const long long p = (long long)((unsigned long long)r - (0x4B400000ull << 24) - (0x4B400000ull << 2) +
                                    (unsigned long long)b1 * 0x1000000ull + (unsigned long long)b2 * 4ull);
    // T (1 + p) in units of 2^-61: T = Th 2^31 + Tl, p = ph 2^32 + pl; the
    // product of the low parts starts at 2^56 so that its sum is not negative
    const long long T = exp_entry(k & (LEAN64_EXP_N - 1));
    const int Th = (int)(T >> 31), Tl = (int)(T & 0x7FFFFFFFll), ph = (int)(p >> 32);
    const unsigned long long V = (unsigned long long)(unsigned)Th * (unsigned)p + 0x0100000000000000ull +
                                 (unsigned long long)((long long)Tl * (ph * 2));
    const long long U = T + (long long)Th * ph + (long long)(V >> 32) - 0x01000000ll;
    // T_0 (1 + p) may lie below 1
    const int low = (int)(U >> 32) < 0x20000000 ? 1 : 0;
    q = (k >> 7) - low;
    return (unsigned long long)U << low;
}

} // namespace detail

// log x with no FP64 instruction.  x = 2^e m, m in [0.707, 1.414) (bin t of
// the top 9 mantissa bits, halved above sqrt 2), c_t ~ 1/m:
//   r = m c - 1 = R 2^-64          exact: one integer product modulo 2^64
//   d = log1p(r) - r               float-float, ~2^-47 relative; r enters as
//                                  rh + rl, the two words of R
//   log x = e ln2 - log c + r + d  64-bit fixed point: 2^-64 for e = 0, 2^-58
//                                  for |e| <= 15, 2^-51 beyond (|log x| >= 2^-9,
//                                  0.34 and 10.7: a few units of 2^-55 relative)
// rounded once to double.  In [1 - 2^-9, 1 + 2^-9) c = 1 and the scale
// follows r (log x = r + d), so log x keeps full relative accuracy at
// x = 1 +- 2^-53.
LEAN64_FN double lean_log(double x) {
    using namespace detail;
    const long long b = d2ll(x);
    const unsigned hi = (unsigned)((unsigned long long)b >> 32);
    // positive, normal and finite?
    if (hi - 0x00100000u >= 0x7FE00000u)
        return log(x);
    const int e = (int)(hi + ((512u - LEAN64_LOG_SPLIT) << 11) - 0x3FF00000u) >> 20;  // bins above the split carry
    const bool near1 = hi - 0x3FEFF000u < 0x1800u;
    const longlong2 ent = log_entry((hi >> 11) & 0x1FFu);  // {c_t, L_t}, one 16-byte load
    const unsigned C = near1 ? (hi < 0x3FF00000u ? 2048u : 4096u) : (unsigned)ent.x;
    const unsigned long long M = ((unsigned long long)((hi & 0x000FFFFFu) | 0x00100000u) << 32) | (unsigned)b;
    const long long R = (long long)(M * C);
    if (near1) {
        if (R == 0)
            return 0.0;
        float dh, dl;
        log_tail(R, dh, dl);
        const unsigned long long A = R < 0 ? 0ull - (unsigned long long)R : (unsigned long long)R;
        const int lz = clz64(A);  // |r| < 2^-9: lz >= 9
        const int F = 62 + lz;
        const long long Sr = (long long)(A << (lz - 2));
        return fix_to_double((R < 0 ? -Sr : Sr) + fix_from_float(dh, F) + fix_from_float(dl, F), F);
    }
    const long long T = log_bin(R, ent.y);
    const int s = e == 0 ? 0 : ((unsigned)(e + 15) <= 30u ? 6 : 13);
    const long long Q = T + (long long)e * (2ll * LEAN64_LN2_L);
    const long long Z = (long long)(int)((unsigned)e << ((33 - s) & 31)) * LEAN64_LN2_H + (Q >> s);
    return fix_wide_to_double(Z, 64 - s);
}

// exp x with no FP64 instruction.  k = round(x 128 / ln2) from a float,
// 2^(k/128) = 2^k' T_j:
//   r = x - k ln2 / 128            64-bit fixed point, 2^-63, modulo 2^64
//   d = expm1(r) - r               float-float, ~2^-47 relative
//   exp x = 2^k' T_j (1 + r + d)   integer products, rounded once
LEAN64_FN double lean_exp(double x) {
    using namespace detail;
    const long long b = d2ll(x);
    const unsigned hi = (unsigned)((unsigned long long)b >> 32), a = hi & 0x7FFFFFFFu;
    if (a >= 0x4085E000u)  // |x| >= 700, inf, NaN
        return exp(x);
    // |x| as a float, cut to 24 bits (2^-126 for what is smaller), with x's sign
    const unsigned am = a > 0x38100000u ? a : 0x38100000u;
    const float xf = u2f((((am << 3) | ((unsigned)b >> 29)) - (896u << 23)) | (hi & 0x80000000u));
    const int k = (int)(f2u(fmaf(xf, (float)LEAN64_INV_LN2N, 12582912.f)) - 0x4B400000u);
    // x in units of 2^-63 modulo 2^64 (the high bits cancel in r; below 2^-11 cut at 2^-63)
    const unsigned long long M = (((unsigned long long)b) & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const int n = (int)(a >> 20) - 1012;  // -1012 .. 20
    const unsigned long long X = n >= 0 ? M << n : M >> (n < -63 ? 63 : -n);
    const unsigned long long sx = (unsigned long long)((long long)(int)hi >> 63);
    int q;
    const unsigned long long m = (exp_bin(k, (long long)((X ^ sx) - sx - k_ln2n(k)), q) + 0x100ull) >> 9;  // leading bit at 52
    return ll2d((long long)(((unsigned long long)(q + 1022) << 52) + m));
}

// 1/b with no FP64 instruction.  b = +-2^E m, m = M 2^-52 in [1, 2);
// y0 = Y 2^-23 ~ 1/m from the MUFU reciprocal; 1 - m y0 = e = -N 2^-75 exactly
// (the product M Y modulo 2^64; |e| < 2^-21); 1/m = y0 (1 + e + e^2) to 2^-62,
// with e and e^2 in units of 2^-60, rounded once; 2^-E and the sign go on the
// bits.  Zero, subnormal, |b| >= 2^1022 (a subnormal result), inf and NaN take
// IEEE 1/b.  a / b is a * lean_rcp(b): one FP64 multiply.
LEAN64_FN double lean_rcp(double b) {
    using namespace detail;
    const unsigned long long bb = (unsigned long long)d2ll(b);
    const unsigned hi = (unsigned)(bb >> 32);
    if ((hi & 0x7FFFFFFFu) - 0x00100000u >= 0x7FC00000u)
        return 1.0 / b;
    const float m1 = u2f((((hi << 3) | ((unsigned)bb >> 29)) & 0x007FFFFFu) | 0x3F800000u);
    const unsigned Y = f2u(fadd(rcp_approx(m1), 1.f)) - 0x3F800000u;  // in (2^22, 2^23]
    const unsigned long long M = ((unsigned long long)((hi & 0x000FFFFFu) | 0x00100000u) << 32) | (unsigned)bb;
    const long long N = (long long)(M * Y);
    const int nh = (int)(N >> 32);
    // -(e + e^2) in units of 2^-60, rounded
    const long long c = (N - (long long)((unsigned long long)((long long)nh * nh) >> 11) + 0x4000ll) >> 15;
    const long long C = (1ll << 29) - c * (long long)Y;  // units of 2^-83, half of 2^-53 added
    const unsigned long long m = (unsigned long long)((C >> 30) + ((long long)Y << 30));  // 1/m in units of 2^-53
    const unsigned mh = (unsigned)(m >> 32) + 0x7FC00000u - (hi & 0xFFF00000u);
    return ll2d((long long)(((unsigned long long)mh << 32) | (unsigned)m));
}

// ---------------------------------------------------------------- fixed point
// Values between elementary functions as 64-bit integers in units of 2^-57
// (|v| < 64): the functions above spend a third of their instructions on
// taking doubles apart and putting them together, and a product or a sum
// between two of them is an FP64 instruction, 16 clocks of its pipe, where 64-bit
// integer sums and products take 1 - 5 of the integer pipes.  The caller
// keeps arguments in range.

// The literal x in units of 2^-F.
__host__ __device__ constexpr long long fx_const(double x, int F = 57) { return (long long)(x * (double)(1ull << F)); }

// a b 2^-F, rounded down: units of 2^-F times another unit.
LEAN64_FN long long fx_mul(long long a, long long b, int F = 57) {
    const unsigned long long lo = (unsigned long long)a * (unsigned long long)b;
    return (long long)(((unsigned long long)detail::mulhi_s64(a, b) << (64 - F)) | (lo >> F));
}

// log x, x positive, normal and finite and |log x| < 64 (else a number modulo
// 128, which no caller uses); |e| / 2 + 2 units for x = 2^e m.
LEAN64_FN long long lean_log_fx(double x) {
    using namespace detail;
    const long long b = d2ll(x);
    const unsigned hi = (unsigned)((unsigned long long)b >> 32);
    const int e = (int)(hi + ((512u - LEAN64_LOG_SPLIT) << 11) - 0x3FF00000u) >> 20;
    const longlong2 ent = log_entry((hi >> 11) & 0x1FFu);
    const unsigned long long M = ((unsigned long long)((hi & 0x000FFFFFu) | 0x00100000u) << 32) | (unsigned)b;
    return (long long)((unsigned long long)(log_bin((long long)(M * (unsigned)ent.x), ent.y) >> 7) +
                       (unsigned long long)(long long)e * LEAN64_LN2_57);
}

// log(N 2^E), N with its leading bit at 63 (taken as its top 53 bits and the
// middle of the rest: 2^-54 relative).
LEAN64_FN long long log_wide_fx(unsigned long long N, int E) {
    using namespace detail;
    const unsigned hi = (unsigned)(N >> 43);  // 1 and 20 mantissa bits
    const longlong2 ent = log_entry((hi >> 11) & 0x1FFu);
    const unsigned C = (unsigned)ent.x;
    const int e = 63 + E + (int)((hi + ((512u - LEAN64_LOG_SPLIT) << 11)) >> 21);
    return (log_bin((long long)((N >> 11) * C + (C >> 1)), ent.y) >> 7) + (long long)e * LEAN64_LN2_57;
}

// log(3 + x), x positive and normal.
LEAN64_FN long long lean_log3p_fx(double x) {
    using namespace detail;
    const unsigned long long b = (unsigned long long)d2ll(x);
    const int ex = (int)(b >> 52) - 1023;
    const unsigned long long B = ((b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << 9;  // 2^-61 at x = 1
    const unsigned long long A = 0x6000000000000000ull;                                       // 3
    const int n = ex < 0 ? -ex : ex, sh = n > 63 ? 63 : n;
    const unsigned long long Y = (ex > 0 ? B : A) + ((ex > 0 ? A : B) >> sh);
    const int lz = clz32((unsigned)(Y >> 32));
    return log_wide_fx(Y << lz, (ex > 0 ? ex : 0) - 61 - lz);
}

// log of a fixed-point value, v > 0.
LEAN64_FN long long log_of_fx(long long v) {
    const int lz = detail::clz64((unsigned long long)v);
    return log_wide_fx((unsigned long long)v << lz, -57 - lz);
}

// exp of a fixed-point value: k and r of lean_exp.
LEAN64_FN unsigned long long exp_fx_bin(long long x, int &q) {
    using namespace detail;
    const int k = (int)(((long long)(int)(x >> 32) * LEAN64_INV_LN2N_22 + (1ll << 46)) >> 47);
    return exp_bin(k, (long long)(((unsigned long long)x << 6) - k_ln2n(k)), q);
}
LEAN64_FN double lean_exp_fx(long long x) {
    int q;
    const unsigned long long m = (exp_fx_bin(x, q) + 0x100ull) >> 9;
    return detail::ll2d((long long)(((unsigned long long)(q + 1022) << 52) + m));
}
// exp x as a fixed-point value, x < log 64.
LEAN64_FN long long exp_to_fx(long long x) {
    int q;
    const unsigned long long U = exp_fx_bin(x, q);  // U 2^(q - 61)
    const int sh = 5 - q;
    return (long long)((U << 1) >> (sh > 63 ? 63 : sh));
}

// 1/m of D = m 2^63 (leading bit at 63) in units of 2^-62, in (2^61, 2^62], to
// about 2^-60: lean_rcp's steps with the residual of all 64 bits.
LEAN64_FN unsigned long long rcp_wide(unsigned long long D) {
    using namespace detail;
    const float m1 = u2f(((unsigned)(D >> 40) & 0x007FFFFFu) | 0x3F800000u);
    const unsigned Y = f2u(fadd(rcp_approx(m1), 1.f)) - 0x3F800000u;
    const long long N = (long long)((D >> 11) * Y) + (long long)((((unsigned)D & 0x7FFu) * (unsigned long long)Y) >> 11);
    const int nh = (int)(N >> 32);
    const long long c = (N - (long long)((unsigned long long)((long long)nh * nh) >> 11) + 0x4000ll) >> 15;
    return (unsigned long long)(((long long)Y << 39) - ((c * (long long)Y) >> 21));
}

// A fixed-point value as a double, |v| >= 2^-25.
LEAN64_FN double from_fx(long long v, int F = 57) { return detail::fix_wide_to_double(v, F); }
// The same for any v (the last bit of the magnitude is lost).
LEAN64_FN double from_fx_any(long long v, int F = 57) {
    const unsigned long long U = (unsigned long long)(v ^ (v >> 63)) | 1ull;
    const int lz = detail::clz64(U) - 1;  // |v| < 2^63
    const unsigned long long m = ((U << lz) + 0x200ull) >> 10;
    return detail::ll2d((long long)((((unsigned long long)(1084 - lz - F) << 52) + m) |
                                    ((unsigned long long)v & 0x8000000000000000ull)));
}

// N / D as a double, 0 < N, D < 2^63 in the same units, to 0.5 ulp and a little.
LEAN64_FN double ratio_fx(unsigned long long N, unsigned long long D) {
    using namespace detail;
    const int ln = clz64(N), ld = clz64(D);
    return fix_wide_to_double((long long)mulhi_u64(N << ln, rcp_wide(D << ld)), 61 - ld + ln);
}

// A double in [0, 1] in units of 2^-62; |x| < 2^(62 - F) in units of 2^-F,
// rounded down in magnitude.
LEAN64_FN unsigned long long unit_to_fx62(double x) {
    const unsigned long long b = (unsigned long long)detail::d2ll(x);
    const int sh = 1023 - (int)(b >> 52);
    const unsigned long long M = ((b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) << 10;
    return M >> (sh > 63 ? 63 : sh);
}
LEAN64_FN long long to_fx(double x, int F) {
    const unsigned long long b = (unsigned long long)detail::d2ll(x);
    const int n = ((int)(b >> 52) & 0x7FF) - 1075 + F;
    const unsigned long long M = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const unsigned long long v = n >= 0 ? M << (n & 63) : M >> (n < -63 ? 63 : -n);
    return (long long)b < 0 ? -(long long)v : (long long)v;
}

// 1 - (1 - x) with both subtractions rounded, 0 < x <= 1: x rounded to a
// multiple of 2^-53 (half to even), on the bits of x.
LEAN64_FN double round_by_one(double x) {
    const unsigned long long b = (unsigned long long)detail::d2ll(x);
    const int sh = 1022 - (int)(b >> 52);  // bits below 2^-53
    if (sh <= 0)
        return x;
    if (sh > 52)
        return sh > 53 || (sh == 53 && (b & 0x000FFFFFFFFFFFFFull) == 0) ? 0.0 : 0x1p-53;
    const unsigned long long unit = 1ull << sh, lsb = (((b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull) >> sh) & 1ull;
    return detail::ll2d((long long)((b + (unit >> 1) - 1ull + lsb) & ~(unit - 1ull)));
}

LEAN64_FN double lean_div(double a, double b) { return a * lean_rcp(b); }

// a / b rounded to nearest, unless it lies within about 2^-52 ulp of a tie:
// Markstein's correction of a rcp(b) by its exact residual (P. Markstein, IBM J.
// Res. Dev. 34(1), 1990; his theorem asks for a correctly rounded reciprocal,
// lean_rcp's is 0.504 ulp), 3 FP64 instructions instead of 8.5.  For |a| and |b| in
// [2^-400, 2^400); everything else takes the hardware's division sequence.
LEAN64_FN bool qdiv_range(double a) {
    return ((unsigned)((unsigned long long)detail::d2ll(a) >> 32) & 0x7FFFFFFFu) - 0x26F00000u < 0x32000000u;
}
LEAN64_FN double qdiv_fast(double a, double b) {
    const double y = lean_rcp(b);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
LEAN64_FN double qdiv(double a, double b) { return qdiv_range(a) && qdiv_range(b) ? qdiv_fast(a, b) : a / b; }

__device__ __forceinline__ double lean_sqrt(double x) {
    const float xf = fpconv::f32(x);
    if (!(xf >= 2e-38f && xf <= 1e38f))
        return sqrt(x);
    const double y = fpconv::f64(rsqrt_approx(xf));
    const double h = 0.5 * y;
    double s = x * y;
    double r = fma(-s, s, x);
    s = fma(r, h, s);
    r = fma(-s, s, x);
    return fma(r, h, s);
}

} // namespace lean64
