"""Generates lean64_tables.h: the lookup tables and constants of the
table-driven FP64 log and exp in lean64.cuh (table methods after
P. T. P. Tang, "Table-driven implementation of the logarithm function in IEEE
floating-point arithmetic", ACM TOMS 16(4), 1990, and "... of the exponential
function ...", ACM TOMS 15(2), 1989).  Values are computed with mpmath at 60
digits and rounded once.

    python noa_gb300/csrc/gen_lean64_tables.py > noa_gb300/csrc/lean64_tables.h
"""
import struct

import mpmath

mpmath.mp.dps = 60

LOG_BITS = 9        # 512 bins over the top 9 mantissa bits
LOG_SPLIT = 212     # bins t >= 212 (m >= 1 + 212/512 > sqrt 2) are halved: m in [0.707, 1)
C_BITS = 11         # c_t = C_t / 2^11
EXP_N = 128         # 2^(j/128)
# a float near these carries an integer in its low bits: 1.5 2^23 one of
# +-2^22, 2^24 - 1 one of -2^23 .. 0
MAGIC = 0x4B400000
MAGIC_NEG = 0x4B7FFFFF


def f32(x):
    return struct.unpack("f", struct.pack("f", float(x)))[0]


def ff(x):
    """x as a float pair h + l (h = x rounded to float, l = the rest)."""
    h = f32(x)
    return h, f32(mpmath.mpf(x) - mpmath.mpf(h))


def log_tables():
    """Per bin t: (c_t 2^12 / 2^h, L_t).

    c_t = C_t / 2^11 is 1 / (bin centre) rounded to 11 fractional bits and
    m = M 2^-(52+h), so that r = m c_t - 1 is an exact multiple of 2^-64: the
    product of the two integers modulo 2^64; |r| < 2^-9.5.  L_t is -log(c_t)
    in units of 2^-64, less the offsets MAGIC_NEG 2^22 and MAGIC that the two
    integer parts of the sum carry, modulo 2^64.
    """
    rows = []
    one = 1 << C_BITS
    for t in range(1 << LOG_BITS):
        h = 1 if t >= LOG_SPLIT else 0
        lo = (1 + mpmath.mpf(t) / (1 << LOG_BITS)) / 2 ** h
        hi = (1 + mpmath.mpf(t + 1) / (1 << LOG_BITS)) / 2 ** h
        C = int(mpmath.nint(one / ((lo + hi) / 2)))
        for m in (lo, hi):  # |r| stays below 2^-9.5 over the bin
            assert abs(m * C / one - 1) < mpmath.mpf(2) ** -9.5
        L = int(mpmath.nint(-mpmath.log(mpmath.mpf(C) / one) * mpmath.mpf(2) ** 64))
        L = (L - (MAGIC_NEG << 22) - MAGIC) % (1 << 64)
        rows.append((C << (1 - h), L - (1 << 64) if L >> 63 else L))
    return rows


def signed_words(v, n):
    """v (an integer) as n words of 32 bits, each in [-2^31, 2^31), lowest first."""
    w = []
    for _ in range(n):
        d = v & 0xFFFFFFFF
        d -= (1 << 32) if d >> 31 else 0
        w.append(d)
        v = (v - d) >> 32
    assert v == 0
    return w


def main():
    rows = log_tables()
    ln2 = mpmath.log(2)
    ln2_l, ln2_h = signed_words(int(mpmath.nint(ln2 * mpmath.mpf(2) ** 63)), 2)  # LN2_L doubles in units of 2^-64
    k_l, k_m, k_h = signed_words(int(mpmath.nint(ln2 / EXP_N * mpmath.mpf(2) ** 95)), 3)
    T = [int(mpmath.nint(mpmath.power(2, mpmath.mpf(j) / EXP_N) * mpmath.mpf(2) ** 61)) for j in range(EXP_N)]
    third_h, third_l = ff(mpmath.mpf(1) / 3)
    sixth_h, sixth_l = ff(mpmath.mpf(1) / 6)
    out = []
    out.append("/* Generated by gen_lean64_tables.py -- do not edit. */")
    out.append("#pragma once")
    out.append(f"#define LEAN64_LOG_BITS {LOG_BITS}")
    out.append(f"#define LEAN64_LOG_SPLIT {LOG_SPLIT}")
    out.append(f"#define LEAN64_EXP_N {EXP_N}")
    out.append(f"#define LEAN64_INV_LN2N {float(EXP_N / ln2)!r}")
    out.append("/* ln 2 = LN2_H 2^-31 + LN2_L 2^-63 */")
    out.append(f"#define LEAN64_LN2_H {ln2_h}")
    out.append(f"#define LEAN64_LN2_L {ln2_l}")
    out.append("/* ln 2 in units of 2^-57 */")
    out.append(f"#define LEAN64_LN2_57 {int(mpmath.nint(ln2 * mpmath.mpf(2) ** 57))}LL")
    out.append("/* 128 / ln 2 in units of 2^-22 */")
    out.append(f"#define LEAN64_INV_LN2N_22 {int(mpmath.nint(EXP_N / ln2 * 2 ** 22))}")
    out.append("/* ln 2 / 128 = K_H 2^-31 + K_M 2^-63 + K_L 2^-95 */")
    out.append(f"#define LEAN64_K_H {k_h}")
    out.append(f"#define LEAN64_K_M {k_m}")
    out.append(f"#define LEAN64_K_L {k_l}")
    out.append(f"#define LEAN64_THIRD_H {third_h!r}f")
    out.append(f"#define LEAN64_THIRD_L {third_l!r}f")
    out.append(f"#define LEAN64_SIXTH_H {sixth_h!r}f")
    out.append(f"#define LEAN64_SIXTH_L {sixth_l!r}f")
    out.append("/* Per bin t, one 16-byte entry {c_t, L_t}: the reciprocal c_t of the bin")
    out.append("   centre in units of 2^-12 (2^-11 for the halved bins t >= LOG_SPLIT; 11")
    out.append("   fractional bits) and -log(c_t) in units of 2^-64, less the offsets of the")
    out.append("   two float-carried integers that are added to it (MAGIC_NEG 2^22 + MAGIC). */")
    out.append("#define LEAN64_LOG_TAB_DATA {\\")
    out.append(",\\\n".join("    {%dLL, %dLL}" % r for r in rows) + "}")
    out.append("static __device__ const longlong2 lean64_log_tab[%d] = LEAN64_LOG_TAB_DATA;" % len(rows))
    out.append("/* 2^(j/128) in units of 2^-61, rounded. */")
    out.append("#define LEAN64_EXP_TAB_DATA {\\")
    out.append(",\\\n".join("    %dLL" % v for v in T) + "}")
    out.append("static __device__ const long long lean64_exp_t[%d] = LEAN64_EXP_TAB_DATA;" % len(T))
    print("\n".join(out))


if __name__ == "__main__":
    main()
