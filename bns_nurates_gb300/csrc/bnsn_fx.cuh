// Double-precision exp, log, pow and Fermi-Dirac integrals on the integer
// pipes.
//
// Why: GB300 issues 2 FP64 lanes per SM and clock, so one FP64 warp
// instruction holds its pipe for 16 clocks, while 32x32-bit multiplies run at
// 64 (wide or high half: 28-31), additions and shifts at ~64-100 lanes.  The
// opacity kernels were bound by that pipe (85-86% busy), most of it spent in
// elementary functions: measured per lane in units of one FP64 FMA, exp 17,
// log 33, pow 100, a division 5-7, the rational Fermi integrals F_1..F_5 150.
// The functions below work on 64-bit fixed-point numbers, which hold 11 bits
// more than a double's mantissa: 2^x and log2 x take ~35 clocks (2.2 FMA) per
// warp and F_1..F_5 ~150 clocks (9 FMA).  Error bounds (tests/test_fx.py measures them on
// the host, the same source compiled by g++): e^x one ulp (2^-52); F_k 2^-51; x^p 2^-52 + |p|
// 2^-55, since log2 x carries 2^-56; log and log2 an absolute 2^-56, so near x = 1 they
// are not relatively accurate; quotients 2^-51.
//
// Methods: table-driven exponential and logarithm (P. T. P. Tang, ACM TOMS 15
// (1989) 144 and 16 (1990) 378) carried out in fixed point; Fermi integrals by
// their Taylor series from a table of the normalised integrals phi_k = F_k / k!
// at multiples of 1/8: d phi_k / dx = phi_{k-1}, so one table row serves all
// orders; the reciprocal is an approximate one with a third-order
// (Halley) correction.
//
// Arguments outside the fixed-point ranges (overflow, underflow, NaN,
// denormals) take the CUDA library function in a rare branch, out of line.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define BNSN_FX_HD __device__ __forceinline__
#define BNSN_FX_OUT static __device__ __noinline__
#define BNSN_FX_TABLE static __device__ const
#else
#define BNSN_FX_HD static inline
#define BNSN_FX_OUT static
#define BNSN_FX_TABLE static const
#endif

#include "bnsn_fx_tab.h"

namespace bnsn {
namespace fx {

#ifdef __CUDACC__
BNSN_FX_HD uint32_t umulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
BNSN_FX_HD int32_t smulhi(int32_t a, int32_t b) { return __mulhi(a, b); }
BNSN_FX_HD uint64_t umul64hi(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
BNSN_FX_HD int clz64(uint64_t a) { return __clzll((long long)a); }
BNSN_FX_HD uint64_t bits_of(double x) { return (uint64_t)__double_as_longlong(x); }
BNSN_FX_HD double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
// ~20-bit reciprocal (one special-function instruction)
BNSN_FX_HD double rcp_approx(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}
#else
BNSN_FX_HD uint32_t umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
BNSN_FX_HD int32_t smulhi(int32_t a, int32_t b) { return (int32_t)(((int64_t)a * b) >> 32); }
BNSN_FX_HD uint64_t umul64hi(uint64_t a, uint64_t b)
{
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
}
BNSN_FX_HD int clz64(uint64_t a) { return __builtin_clzll(a); }
BNSN_FX_HD uint64_t bits_of(double x)
{
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
}
BNSN_FX_HD double from_bits(uint64_t b)
{
    double x;
    memcpy(&x, &b, 8);
    return x;
}
BNSN_FX_HD double rcp_approx(double x) // the device's precision
{
    return from_bits(bits_of(1. / x) & 0xffffffff00000000ull);
}
#endif

// a * b / 2^64, up to 3 units low (the product of the low words is dropped).
BNSN_FX_HD uint64_t mulhi3(uint64_t a, uint64_t b)
{
    const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a;
    const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
    return (uint64_t)ah * bh + umulhi(ah, bl) + umulhi(al, bh);
}

// The same for signed a and b < 2^63.
BNSN_FX_HD int64_t mulhi3s(int64_t a, uint64_t b)
{
    const int32_t ah  = (int32_t)(a >> 32);
    const uint32_t al = (uint32_t)a, bl = (uint32_t)b;
    const int32_t bh  = (int32_t)(b >> 32);
    const int32_t m   = (int32_t)(umulhi((uint32_t)ah, bl) - (ah < 0 ? bl : 0u));
    return (int64_t)ah * bh + m + umulhi(al, (uint32_t)bh);
}

// 1/x to about half an ulp for x and 1/x in the normal range.
BNSN_FX_HD double rcp(double x)
{
    const double r = rcp_approx(x);
    const double e = fma(-x, r, 1.);
    return fma(r, fma(e, e, e), r);
}

// a/b to about one ulp (b and 1/b in the normal range).
BNSN_FX_HD double quot(double a, double b)
{
    const double r = rcp(b), q = a * r;
    return fma(fma(-b, q, a), r, q);
}

// x in [2^-400, 2^400)
BNSN_FX_HD bool mid_range(double x)
{
    return (((uint32_t)(bits_of(x) >> 52) & 0x7ffu) - (1023u - 400u)) < 800u;
}

BNSN_FX_OUT double div_special(double a, double b) { return a / b; }

// a/b for any a and b.
BNSN_FX_HD double div(double a, double b)
{
    return mid_range(a) && mid_range(b) ? quot(a, b) : div_special(a, b);
}

// An exponent of two, I + F / 2^64.
struct Exp2
{
    int I;
    uint64_t F;
};

// -(I + F)
BNSN_FX_HD Exp2 negate(Exp2 x)
{
    x.I = x.F ? ~x.I : -x.I;
    x.F = 0ull - x.F;
    return x;
}

// 2^(I + F) for -1022 <= I <= 1022.
BNSN_FX_HD double exp2(Exp2 x)
{
    const int I      = x.I;
    const uint32_t j = (uint32_t)(x.F >> 57);
    const uint64_t R = x.F << 7; // remainder < 2^-7, times 2^71
    const uint64_t T = kExp2[j];
    // u = r ln 2; U = u 2^71
    const uint64_t U  = mulhi3(R, 0xB17217F7D1CF79ABull);
    const uint32_t vh = (uint32_t)(U >> 32);
    // e^u - 1 = u (1 + g), g = (u/2)(1 + k), k = u/3 + u^2/12 + u^3/60 + u^4/360;
    // K = k 2^41
    uint32_t K = 17476u + umulhi(23u, vh);
    K          = 11184811u + umulhi(K, vh);
    K          = 1431655765u + umulhi(K, vh);
    K          = vh + umulhi(K, vh);
    const uint64_t G =
        U + (((uint64_t)(uint32_t)(U >> 32) * K + umulhi((uint32_t)U, K)) >> 9); // g 2^72
    const uint64_t Q = U + (mulhi3(U, G) >> 8);                                   // (e^u - 1) 2^71
    const uint64_t V = T + (mulhi3(T, Q) >> 7);                                   // [1, 2) 2^63
    const uint64_t m = (V >> 11) + ((V >> 10) & 1u);
    return from_bits(m + ((uint64_t)(uint32_t)(I + 1022) << 52));
}

// x log2(e) for |x| < 709.
BNSN_FX_HD Exp2 exp_arg(double x)
{
    const uint64_t b = bits_of(x);
    const int e      = (int)((b >> 52) & 0x7ffu) - 1023; // <= 9
    const uint64_t M = (b << 11) | 0x8000000000000000ull;
    const uint64_t P = umul64hi(M, 0xB8AA3B295C17F0BCull); // |x| log2(e) 2^(62 - e)
    Exp2 r;
    if (e >= -2)
    {
        r.I = (int)(P >> (62 - e < 63 ? 62 - e : 63)) & (e >= -1 ? -1 : 0);
        r.F = P << (2 + e);
    }
    else
    {
        r.I = 0;
        r.F = -2 - e > 63 ? 0ull : P >> (-2 - e);
    }
    return (int64_t)b < 0 ? negate(r) : r;
}

BNSN_FX_OUT double exp_special(double x) { return ::exp(x); }

// e^x for any x.
BNSN_FX_HD double exp(double x)
{
    if (((uint32_t)(bits_of(x) >> 32) & 0x7fffffffu) >= 0x40862000u) // |x| >= 708 or NaN
        return x < -746. ? 0. : exp_special(x);
    return exp2(exp_arg(x));
}

// log2(x) 2^56 (rounded) for x in [2^-120, 2^120].
BNSN_FX_HD int64_t log2_q56(double x)
{
    const uint64_t b  = bits_of(x);
    const int e       = (int)(b >> 52) - 1023;
    const uint64_t M  = (b & 0xfffffffffffffull) | 0x10000000000000ull;
    const LogRow row  = kLog[(uint32_t)(b >> 45) & 127u];
    const int64_t Z   = (int64_t)(M * row.c - 0x8000000000000000ull); // z 2^63, |z| < 2^-7.9
    const int64_t Zn  = Z * 128;                                      // z 2^70
    const uint64_t az = (uint64_t)(Zn < 0 ? -Zn : Zn);
    const uint64_t S  = mulhi3(az, az); // z^2 2^76
    // ln(1 + z) = z - z^2 (1/2 + w), w = -z/3 + v, v = z^2 (1/4 - z/5 + z^2/6)
    const int32_t z32 = (int32_t)(Zn >> 32); // z 2^38
    int32_t t         = 2 * smulhi(43691, z32) - 6710886;
    t                 = 1073741824 + 2 * smulhi(t, z32);
    const int64_t V   = (int64_t)(int32_t)(S >> 32) * t;                        // v 2^76
    const int64_t w   = (V >> 6) - mulhi3s(Zn, 0x5555555555555556ull);          // w 2^70
    const int64_t C   = (int64_t)(S >> 1) + (mulhi3s(w, S) >> 6);               // 2^76
    const int64_t N   = Z - (C >> 13);                                    // ln(1 + z) 2^63
    const int64_t N2  = N + mulhi3s(N, 0x71547652B82FE177ull);            // x log2(e)
    return ((int64_t)e << 56) + (((int64_t)row.l + N2 + 64) >> 7);
}

BNSN_FX_OUT double pow_special(double x, double p) { return ::pow(x, p); }
BNSN_FX_OUT double log_special(double x) { return ::log(x); }

// The exponent p as p 2^58 (|p| < 31.9).
BNSN_FX_HD int64_t pow_exponent(double p) { return (int64_t)(p * 288230376151711744.); }

// p log2(x) from L = log2(x) 2^56 and P = p 2^58, clamped to +-1021.
BNSN_FX_HD Exp2 scale_log(int64_t L, int64_t P)
{
    const uint64_t aL = (uint64_t)(L < 0 ? -L : L), aP = (uint64_t)(P < 0 ? -P : P);
    const uint64_t hi = umul64hi(aL, aP), lo = aL * aP; // 2^114
    Exp2 r;
    r.I = (int)(hi >> 50);
    r.F = (hi << 14) | (lo >> 50);
    if (r.I >= 1021)
    {
        r.I = 1021;
        r.F = 0ull;
    }
    return (L < 0) != (P < 0) ? negate(r) : r;
}

// x^p from log2(x) 2^56 and p 2^58.
BNSN_FX_HD double pow_q(int64_t L, int64_t P) { return exp2(scale_log(L, P)); }

// x in [2^-120, 2^120]
BNSN_FX_HD bool log2_range(double x)
{
    return ((uint32_t)(bits_of(x) >> 52) - (1023u - 120u)) < 240u;
}

// log2(x) and log(x) for any x, to an absolute 2^-56: not relatively accurate near x = 1
// (log(1 + 2^-30) holds 28 bits).
BNSN_FX_HD double log2(double x)
{
    return log2_range(x) ? (double)log2_q56(x) * 1.3877787807814457e-17
                         : log_special(x) * 1.4426950408889634;
}
BNSN_FX_HD double log(double x)
{
    return log2_range(x) ? (double)log2_q56(x) * (0.693147180559945309 * 1.3877787807814457e-17) : log_special(x);
}

// x^p for any x and p.
BNSN_FX_HD double pow(double x, double p)
{
    if (!log2_range(x) || !(fabs(p) < 31.9))
        return pow_special(x, p);
    const Exp2 E = scale_log(log2_q56(x), pow_exponent(p));
    if (E.I >= 1021 || E.I <= -1021)
        return pow_special(x, p);
    return exp2(E);
}

// ---------------------------------------------------------------------------
// Fermi-Dirac integrals F_k(y), k = KLO..KHI (0 <= KLO, KHI <= 5), the
// reference's unnormalised ones (functions.hpp:1550-2838); out[k - KLO].
// A NaN argument yields 0, as the reference's regime tests do.
//
// phi_k(y0 + h) = sum_j phi_{k-j}(y0) h^j / j!, 0 <= h < 1/8, in Horner form
// with the products by h / j: five in 64 bits, the rest (2^-27 of the sum and
// less) in 32.  The row's entries carry 2^(s + (5 - m) d), so h is taken
// as h 2^-d.  Above y = 36 the integral equals its polynomial part to
// 2^-60, below -36 it is k! e^y.
// ---------------------------------------------------------------------------

// The polynomial part of F_K at y > 0 (F_K(y) -+ F_K(-y)).
template <int K>
BNSN_FX_HD double fd_poly(double y)
{
    const double y2 = y * y;
    if (K == 0)
        return y;
    if (K == 1)
        return 1.64493406684822644 + 0.5 * y2;
    if (K == 2)
        return y * (3.28986813369645287 + 0.333333333333333333 * y2);
    if (K == 3)
        return 11.3643939539669510 + y2 * (4.93480220054467931 + y2 * 0.25);
    if (K == 4)
        return y * (45.4575758158678040 + y2 * (6.57973626739290575 + y2 * 0.2));
    return 236.532261911384425 +
           y2 * (113.643939539669510 + y2 * (8.22467033424113218 + y2 * 0.166666666666666667));
}

template <int K>
BNSN_FX_HD constexpr double fd_factorial()
{
    return K < 2 ? 1. : K == 2 ? 2. : K == 3 ? 6. : K == 4 ? 24. : 120.;
}

// Entry m of a row in 32 bits (units of 2^32).
template <int M>
BNSN_FX_HD int32_t fd_t(const FdRow& r)
{
    return M >= -5 ? (int32_t)(r.c[M >= -5 ? 5 - M : 0] >> 32) : r.t[M >= -5 ? 0 : -6 - M];
}

// h / j in units of 2^-64 (j = 1..5) and 2^-32 (j = 6..10)
struct FdStep
{
    uint64_t h1, h2, h3, h4, h5;
    int32_t h6, h7, h8, h9, h10;
};

template <int M>
BNSN_FX_HD int64_t fd_mul(int64_t T, uint64_t h) // T: the partial sum from entry M down
{
    return M <= -2 ? mulhi3s(T, h) : (int64_t)mulhi3((uint64_t)T, h);
}

template <int K, bool NORM>
BNSN_FX_HD double fd_one(const FdRow& r, const FdStep& S, int scale, int d)
{
    int32_t t = fd_t<K - 10>(r);
    t         = fd_t<K - 9>(r) + smulhi(t, S.h10);
    t         = fd_t<K - 8>(r) + smulhi(t, S.h9);
    t         = fd_t<K - 7>(r) + smulhi(t, S.h8);
    t         = fd_t<K - 6>(r) + smulhi(t, S.h7);
    int64_t T = r.c[10 - K] + (int64_t)t * S.h6;
    T         = r.c[9 - K] + fd_mul<K - 5>(T, S.h5);
    T         = r.c[8 - K] + fd_mul<K - 4>(T, S.h4);
    T         = r.c[7 - K] + fd_mul<K - 3>(T, S.h3);
    T         = r.c[6 - K] + fd_mul<K - 2>(T, S.h2);
    uint64_t V = (uint64_t)(r.c[5 - K] + fd_mul<K - 1>(T, S.h1));
    // x k!: 2 = 2, 6 = 1.5 x 4, 24 = 1.5 x 16, 120 = 1.875 x 64
    if (!NORM && (K == 3 || K == 4))
        V += V >> 1;
    if (!NORM && K == 5)
        V = 2 * V - (V >> 3);
    constexpr int kExp = NORM || K < 2 ? 0 : K == 2 ? 1 : K == 3 ? 2 : K == 4 ? 4 : 6;
    const int lz       = clz64(V);
    const uint64_t N   = V << lz;
    const uint64_t m   = (N >> 11) + ((N >> 10) & 1u);
    const int e        = 1022 + 63 + kExp - lz - scale - (5 - K) * d;
    return from_bits(m + ((uint64_t)(uint32_t)e << 52));
}

// NORM: phi_k = F_k / k! instead.
template <int KLO, int KHI, bool NORM = false>
BNSN_FX_HD void fd_orders(double y, double* out)
{
    const uint64_t b = bits_of(y);
    const uint32_t a = (uint32_t)(b >> 32) & 0x7fffffffu;
    if (a >= 0x40420000u) // |y| >= 36 or NaN
    {
        if (y > 0.)
        {
#define BNSN_FX_ORDER(K)                                                                           \
    if (KLO <= K && K <= KHI)                                                                      \
        out[K - KLO < 0 ? 0 : K - KLO] =                                                           \
            fd_poly<K>(y) * (NORM ? 1. / fd_factorial<K>() : 1.);
            BNSN_FX_ORDER(0) BNSN_FX_ORDER(1) BNSN_FX_ORDER(2)
            BNSN_FX_ORDER(3) BNSN_FX_ORDER(4) BNSN_FX_ORDER(5)
#undef BNSN_FX_ORDER
        }
        else
        {
            const double ex = y < 0. ? exp(y) : 0.;
#define BNSN_FX_ORDER(K)                                                                           \
    if (KLO <= K && K <= KHI)                                                                      \
        out[K - KLO < 0 ? 0 : K - KLO] = (NORM ? 1. : fd_factorial<K>()) * ex;
            BNSN_FX_ORDER(0) BNSN_FX_ORDER(1) BNSN_FX_ORDER(2)
            BNSN_FX_ORDER(3) BNSN_FX_ORDER(4) BNSN_FX_ORDER(5)
#undef BNSN_FX_ORDER
        }
        return;
    }
    // Y = y 2^57 (truncated), row floor(8 y), h = y - floor(8 y) / 8
    const int sh     = 5 + 1023 - (int)(a >> 20);
    const uint64_t M = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;
    const uint64_t A = sh > 63 ? 0ull : M >> sh;
    const int64_t Y  = (int64_t)b < 0 ? -(int64_t)A : (int64_t)A;
    const int i      = (int)(Y >> 54) + kFdLimit;
    const FdRow& r   = kFdRows[i];
    const int d = r.meta & 255, scale = r.meta >> 8;
    FdStep S;
    S.h1 = (((uint64_t)Y << 10) >> 3) >> d;
    S.h2 = S.h1 >> 1;
    S.h3 = mulhi3(S.h1, 0x5555555555555556ull);
    S.h4 = S.h1 >> 2;
    S.h5 = mulhi3(S.h1, 0x3333333333333334ull);
    const uint32_t h = (uint32_t)(S.h1 >> 32);
    S.h6  = (int32_t)umulhi(h, 715827883u);
    S.h7  = (int32_t)umulhi(h, 613566757u);
    S.h8  = (int32_t)(h >> 3);
    S.h9  = (int32_t)umulhi(h, 477218589u);
    S.h10 = (int32_t)umulhi(h, 429496730u);
#define BNSN_FX_ORDER(K)                                                                           \
    if (KLO <= K && K <= KHI)                                                                      \
        out[K - KLO < 0 ? 0 : K - KLO] = fd_one<K, NORM>(r, S, scale, d);
    BNSN_FX_ORDER(0) BNSN_FX_ORDER(1) BNSN_FX_ORDER(2)
    BNSN_FX_ORDER(3) BNSN_FX_ORDER(4) BNSN_FX_ORDER(5)
#undef BNSN_FX_ORDER
}

// The interval of x in [-4, 100) among those of the Fermi-Dirac family (fdi.cu): 64 of width
// 11/16 below 40, then 6 of width 10; the position in it, in [-1, 1), is returned.
BNSN_FX_HD double fd_interval(double x, int* interval)
{
    const uint64_t bits = bits_of(x), mag = bits & 0x7fffffffffffffffull;
    // y = x + 4 in 2^-56 (exact for |x| >= 1/8), its interval in sixteenths
    const int sh     = 7 + 1023 - (int)(mag >> 52);
    const uint64_t A = sh > 63 ? 0ull : ((mag << 11) | 0x8000000000000000ull) >> sh;
    const int64_t Y  = (4ll << 56) + ((int64_t)bits < 0 ? -(int64_t)A : (int64_t)A);
    const int y16    = (int)(Y >> 52);
    const bool wide  = y16 >= 704;
    const int i      = wide ? (y16 - 704) / 160 : y16 / 11;
    const int w = wide ? 160 : 11, base = wide ? 704 + i * 160 : i * 11;
    *interval = i + (wide ? 64 : 0);
    // 2 (y - start) - width over the width
    const int64_t r = 2 * (Y - ((int64_t)base << 52)) - ((int64_t)w << 52);
    return (double)r * (wide ? 0x1p-52 / 160. : 0x1p-52 / 11.);
}

} // namespace fx
} // namespace bnsn
