// Mixed-precision device helpers shared by the grey and spectral kernels.
#pragma once

#include "bnsn_df.cuh"
#include "bnsn_fp64.cuh"
#include "bnsn_internal.h"

namespace bnsn {
namespace {

using namespace fp64;

// Bracket of lw on a log-w axis of d3 entries (binary search, first interval).
template <class R>
__device__ __forceinline__ int bracket_sorted(R lw, const R* ax, int d3, R* t)
{
    int lo = 0, hi = d3 - 2;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (lw <= ax[mid + 1])
            hi = mid;
        else
            lo = mid + 1;
    }
    *t = (lw - ax[lo]) / (ax[lo + 1] - ax[lo]);
    return lo;
}

// Order-preserving integer image of a double (comparisons off the FP64 pipe).
__device__ __forceinline__ int64_t order_key(double v)
{
    const int64_t b = __double_as_longlong(v);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ Gp19Table gp19_table(const OpacityLaunch& L)
{
    return {L.gp19.d0, L.gp19.d1, L.gp19.d2,    L.gp19.d3,   L.gp19.nb,  L.gp19.ye,
            L.gp19.t,  L.gp19.w,  L.gp19.lognb, L.gp19.logw, L.gp19.data};
}

// The GP19 log w axis in shared memory: values, their order_key and the inverse
// intervals.
struct Gp19Axis
{
    double lw[kGp19MaxW], idl[kGp19MaxW];
    int64_t key[kGp19MaxW];
};

__device__ __forceinline__ void gp19_axis_entry(Gp19Axis& A, const double* logw, int d3, int k)
{
    A.lw[k]  = logw[k];
    A.key[k] = order_key(logw[k]);
    A.idl[k] = k + 1 < d3 ? 1. / (logw[k + 1] - logw[k]) : 0.;
}

// GP19 absorption kernel at w (clipped to the axis) from a point's profiles.
__device__ __forceinline__ double gp19_profile_absorption(const Gp19Point& pt,
                                                          const double (*p)[kGp19MaxW],
                                                          const Gp19Axis& A, int d3, double w)
{
    const double lw = fx::log(w);
    const int64_t k = order_key(lw);
    // smallest l in [0, d3 - 2] with lw <= axis[l + 1]
    int lo = 0, hi = d3 - 2;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (k <= A.key[mid + 1])
            hi = mid;
        else
            lo = mid + 1;
    }
    const double tw = (lw - A.lw[lo]) * A.idl[lo], t0 = 1. - tw;
    const double v0 = fma(p[0][lo + 1], tw, p[0][lo] * t0);
    const double v1 = pt.regime >= 2 ? fma(p[1][lo + 1], tw, p[1][lo] * t0) : 0.;
    return gp19_absorption(pt, v0, v1, w);
}

// One species' occupation constants (distribution.hpp:298-315) for x = omega / u:
// g = wt / (1 + e^{x rt - eta}) + kf x^cf e^{-x rf}.
struct Occ64
{
    double rt, eta, rf, wt, kf, cf;
};

// The degeneracy for it; the reference's argument (omega - T eta) / T is NaN at T = inf.
__device__ __forceinline__ double occ64_eta(const Distr& d, int s)
{
    return isinf(d.temp_t[s]) ? __longlong_as_double(0x7ff8000000000000LL) : d.eta_t[s];
}

__device__ __forceinline__ void occ64_from(const Distr& d, int s, double u, Occ64* o)
{
    o->rt  = u / d.temp_t[s];
    o->eta = occ64_eta(d, s);
    o->rf  = u / d.temp_f[s];
    o->wt  = d.w_t[s];
    o->cf  = d.c_f[s];
    o->kf  = d.w_f[s] * (u == 1. ? d.beta_f[s] : d.beta_f[s] * fx::pow(u, d.c_f[s]));
}

// One species at x, p = x^cf.
__device__ __forceinline__ double occ64_one(const Occ64& o, double x, double p)
{
    const double ft = fx::rcp(safe_exp(fma(x, o.rt, -o.eta)) + 1.);
    return fma(o.wt, ft, o.kf * (p * fx::exp(-x * o.rf)));
}

// Four species at x; xc = x^c0, common: every cf is c0.
__device__ __forceinline__ void occ64_eval(const Occ64* o, double x, double xc, bool common,
                                           double* g)
{
#pragma unroll
    for (int s = 0; s < 4; ++s)
        g[s] = occ64_one(o[s], x, common ? xc : fx::pow(x, o[s].cf));
}

// Heavy-lepton neutrinos and antineutrinos evolved as one species: their
// occupations are the same.
__device__ __forceinline__ bool species_twins(const Distr& d)
{
    return d.w_t[2] == d.w_t[3] && d.temp_t[2] == d.temp_t[3] && d.eta_t[2] == d.eta_t[3] &&
           d.w_f[2] == d.w_f[3] && d.temp_f[2] == d.temp_f[3] && d.c_f[2] == d.c_f[3] &&
           d.beta_f[2] == d.beta_f[3];
}

// 15 y^2 z^2 Psi_0(y, z) and Psi_0(z, y) (kernel_pair.hpp:16-120) from Fermi
// integrals scaled as Psi needs them (pair_scale): am, ap at eta -+ y, bm, bp at
// eta -+ z; f40, f20 = 40 F_3(eta), 20 F_4(eta).  The sums are in the reference's
// order: they cancel, and another order of c10 alone moves ill-conditioned
// outputs by more than the reference's own rounding does.
__device__ __forceinline__ void pair_psi_scaled(const double* am, const double* ap,
                                                const double* bm, const double* bp, double eta,
                                                double y, double z, double f40, double f20,
                                                double* p0, double* p1)
{
    double fm[3], fp[3];
    fdi_orders<3, 5>(eta - y - z, fm);
    fdi_orders<3, 5>(eta + y + z, fp);
    const double c5 = fma(40., fm[0], -f40), c7 = fma(20., fm[1], -f20);
    const double c8 = fma(-40., fp[0], f40), c9 = fma(20., fp[1], -f20);
    const double c10 = fma(-4., fp[2], fma(4., fm[2], -am[4]) - bm[4] + ap[4]) + bp[4];
    const double d01 = bp[3] - am[3], c2 = am[1] - bp[1], c3 = bp[2] - am[2];
    const double d11 = bm[3] - ap[3], c14 = bm[1] - ap[1], c13 = ap[2] - bm[2];
    const double u0 = fma(z, fma(z, bp[0] - am[0], c2), c3 + c5);
    const double v0 = fma(z, fma(-c2, z, -2. * c3), fma(y, u0, d01 + c7));
    *p0 = fma(z, fma(z, c3 + c8, c9 - d01), fma(y, v0, c10));
    const double u1 = fma(y, fma(y, ap[0] - bm[0], c14), c13 + c5);
    const double v1 = fma(z, u1, fma(y, fma(-c14, y, -2. * c13), c7 - d11));
    *p1 = fma(z, v1, fma(y, fma(y, c13 + c8, d11 + c9), c10));
}

// F_1..F_5 scaled for it: 120 F_1, 120 F_2, 40 F_3, 20 F_4, 4 F_5.
__device__ __forceinline__ void pair_scale(const double* f, double* o)
{
    o[0] = 120. * f[0];
    o[1] = 120. * f[1];
    o[2] = 40. * f[2];
    o[3] = 20. * f[3];
    o[4] = 4. * f[4];
}

// The NES/NPS bracket of one lepton at energies x > y (in units of T, dl = x - y):
// MezzacappaIntOut = +-(24 / P^2) (b1 A + b2 B) with P = x y, + for w = x (scattering
// down).  With phi_k = F_k / k!, D_k = phi_k(eta - x) - phi_k(eta - y), E_k =
// phi_k(eta) - phi_k(eta - dl), S = x + y:
//   A = (E5 + D5) + x (E4 + x E3 / 2) + S (D4 + S D3 / 2 + P D2 / 2) + P^2 D1 / 4,
//   B = (E5 + D5) + y (y E3 / 2 - E4).
// fx, fy: phi_1..phi_5 at eta - x, eta - y; fe: F_0..F_5 at eta.
__device__ __forceinline__ void nes_bracket(double eta, double x, double y, double dl,
                                            const double* fx5, const double* fy5,
                                            const double* fe, double* A, double* B)
{
    double f[3];
    fx::fd_orders<3, 5, true>(eta - dl, f);
    const double sm = x + y, hp = 0.5 * (x * y), qp = hp * hp; // P^2 / 4
    const double E3 = fma(fe[3], 0.5 / 6., -0.5 * f[0]);       // E_3 / 2
    const double E4 = fma(fe[4], 1. / 24., -f[1]);
    const double ED = fma(fe[5], 1. / 120., -f[2]) + (fx5[4] - fy5[4]);
    double a = fma(x, fma(x, E3, E4), ED);
    a = fma(sm, fma(hp, fx5[1] - fy5[1], fma(0.5 * sm, fx5[2] - fy5[2], fx5[3] - fy5[3])), a);
    *A = fma(qp, fx5[0] - fy5[0], a);
    *B = fma(y, fma(y, E3, -E4), ED);
}

// The reference's Taylor branches (kernel_nes.hpp:82-132, y <= 10^-3 eta) in the
// same units; fd0 = FermiDistr(0, 1, eta).
__device__ __forceinline__ void nes_bracket_taylor(double eta, double x, double y, double dl,
                                                   const double* fe, double fd0, double* A,
                                                   double* B)
{
    const double hp = 0.5 * (x * y), y2 = y * y, xy = x * y, x2 = x * x;
    const double c  = hp * hp * y * (-1. / 6.) * fx::rcp(x2);
    if (x > eta * 1e-3)
    {
        double f[3];
        fdi_orders<0, 2>(eta - x, f);
        const double f0 = f[2] - fe[2], f1 = f[1], f2 = fe[1];
        const double f3 = f[0] + y * fermi_distr(0., 1., eta - x) * (1. / 6.);
        const double f4 = fe[0] - y * fd0 * (1. / 6.);
        *A = c * (2. * f0 + (y + 4. * x) * f1 + (3. * y - 4. * x) * f2 +
                  (0.2 * y2 + xy + 2. * x2) * f3 - (1.2 * y2 - 3. * xy + 2. * x2) * f4);
        *B = c * (2. * f0 + 3. * y * f1 + y * f2 + 1.2 * y2 * f3 - 0.2 * y2 * f4);
    }
    else
    {
        const double u = 4. * fe[1] + fd0 * (11. * y2 - 25. * xy + 20. * x2) * (1. / 30.);
        const double v = (2. * x - y) * fe[0];
        *A = -dl * c * (u + v);
        *B = -dl * c * (u - v);
    }
}

// Interval of w on the GP19 w axis and its interpolation weight in FP32, for
// an FP64 w already clipped to the axis.  The interval comes from an FP32
// search of log w; the weight from log1p of the offset to the interval's first
// node, (w - w_l) / w_l, so that it keeps the relative precision of that
// offset: logf(w) itself is off by up to an ulp of log w (~5e-7 at w ~ 400
// MeV), which moved the weight by 1e-6 and the brem cell by up to 1.4e-6.
// wax, iw: the axis and 1 / axis (FP64); lwf: log axis (FP32); idl:
// 1 / (log w_{l+1} - log w_l) (FP32).
__device__ __forceinline__ int gp19_bracket32(double w, const float* lwf, const double* wax,
                                              const double* iw, const float* idl, int d3,
                                              float* tw)
{
    float t;
    const int l = bracket_sorted<float>(logf((float)w), lwf, d3, &t);
    *tw         = log1pf((float)((w - wax[l]) * iw[l])) * idl[l];
    return l;
}

// NEPSExpFunc (functions.hpp:4401-4413) in FP32 for the FP64 argument d;
// e^{-|d|} takes the FP32 exponential of the rounded argument times the
// first-order correction for its remainder, expm1 keeps 1 - e^{-|d|}
// accurate for small |d|.
__device__ __forceinline__ float neps_exp_f32(double d, bool neg)
{
    const double ad = fabs(d);
    const float a   = (float)ad;
    const float alo = (float)(ad - (double)a); // e^{-alo} = 1 - alo to FP32 precision
    const float ea  = expf(-a);
    const float e   = ea * (1.f - alo);
    const float dn  = -expm1f(-a) + ea * alo + (d == 0. ? 1.f : 0.f);
    return (neg ? 1.f : -e) / dn;
}

// Taylor branches of neps_pair (kernel_nes.hpp:82-132) for w or w' near 0,
// in FP64: dimensionless r1 = R(w, w'), r2 = R(w', w) of lepton e.  Rare in the
// item loop, so kept out of line to keep the loop's code small.
__device__ __noinline__ void neps_taylor(const NepsPoint& P, int e, double w, double wp,
                                         double x, double y, int sign1, int sign2, double* r1,
                                         double* r2)
{
    const double eta  = e ? P.eta1 : P.eta0;
    const double* f0e = e ? P.fe1 : P.fe0;
    const double fd0  = e ? P.fd01 : P.fd00;
    if (x > eta * 1e-3)
    {
        double fx[3];
        fdi_orders<0, 2>(eta - x, fx);
        const double f[5] = {fx[2] - f0e[2], fx[1], f0e[1],
                             fx[0] + y * fermi_distr(0., 1., eta - x) / 6., f0e[0] - y * fd0 / 6.};
#pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            double b1, b2;
            neps_couplings(e, s, &b1, &b2);
            r1[s] = mb_int_one(x, y, sign1, b1, b2, f);
            r2[s] = mb_int_one(x, y, sign2, b1, b2, f);
        }
    }
    else
    {
        const double f[3] = {fd0, f0e[0], f0e[1]};
#pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            double b1, b2;
            neps_couplings(e, s, &b1, &b2);
            r1[s] = mb_int_two(w, wp, x, y, b1, b2, f);
            r2[s] = mb_int_two(wp, w, x, y, b1, b2, f);
        }
    }
}

} // namespace
} // namespace bnsn

namespace bnsn {
namespace {

// Spectral NES/NPS kernel of one direction before the detailed-balance factors:
// R[s] = sum over e-, e+ of R(w, w') for species s, dimensionless (the caller
// applies the NEPS prefactor, NEPSExpFunc and the occupations), the FP64 bracket
// of each lepton rounded to FP32.  fw[e]: phi_1..phi_5 at eta_e - w.
__device__ __forceinline__ void neps_r_mixed(const NepsPoint& P, double w, double wp,
                                             const double (*fw)[5], float* R)
{
    const bool down  = w > wp;
    const double x   = down ? w : wp, y = down ? wp : w, dl = x - y;
    const double xy  = w * wp;
    const double sc  = (down ? 24. : -24.) * fx::rcp(xy * xy);
    const int nlep   = P.eta0 > 30. ? 1 : 2; // e+ terms below 1e-13 of e- for eta_e > 30
#pragma unroll
    for (int s = 0; s < 4; ++s)
        R[s] = 0.f;
#pragma unroll 1
    for (int e = 0; e < nlep; ++e)
    {
        const double eta = e ? P.eta1 : P.eta0;
        const double* fe = e ? P.fe1 : P.fe0;
        double A, B;
        if (y > eta * 1e-3)
        {
            double fp[5];
            fx::fd_orders<1, 5, true>(eta - wp, fp);
            nes_bracket(eta, x, y, dl, down ? fw[e] : fp, down ? fp : fw[e], fe, &A, &B);
        }
        else
            nes_bracket_taylor(eta, x, y, dl, fe, e ? P.fd01 : P.fd00, &A, &B);
        A *= sc;
        B *= sc;
        constexpr double bp = k::NepsBPlus, bm = k::NepsBMinus, bz = k::NepsBZero;
        const double U = e ? B : A, V = e ? A : B;
        R[0] += (float)fma(bp, U, bz * V);
        R[1] += (float)fma(bp, V, bz * U);
        R[2] += (float)fma(bm, U, bz * V);
        R[3] += (float)fma(bm, V, bz * U);
    }
}

// What neps_r_df needs of a point: eta and the unreflected F_1..F_5 of e- and e+.
struct alignas(8) NesDf
{
    dfm::df reta[2][5], eta[2];
};

// The same with the Fermi integrals and brackets in double-float, for energies nu/T
// below kSpecNesDfW: the brackets difference their integrals over (w w')^2, so there
// the low bits of the integrals show in R (1e-7 at nu/T = 0.05, 4e-9 at 0.2), and
// these are the ones such outputs have always had.  rw[e]: the unreflected F_1..F_5
// at eta_e - w; W, WP are w, wp in df.
__device__ __forceinline__ void neps_r_df(const NepsPoint& P, const NesDf& Q,
                                       const dfm::FdiTab* ftab, double w, double wp, dfm::df W,
                                       dfm::df WP, const dfm::df (*rw)[5], float* R)
{
    using namespace dfm;
    const double x = (w > wp) ? w : wp;
    const double y = (w < wp) ? w : wp;
    const bool n1     = w > wp; // sign of wp - w
    const float sign1 = n1 ? 1.f : -1.f;
#pragma unroll
    for (int s = 0; s < 4; ++s)
        R[s] = 0.f;
    const df S = add(W, WP), Pp = mul(W, WP), Dn = mul(Pp, Pp);
    const df X = n1 ? W : WP, Y = n1 ? WP : W;
    // bracket arguments from FP64 differences (eta up to ~1e3 needs 53 bits)
    const double dd = w - wp, ad = fabs(dd);
    const df dlt    = from_double(dd);    // w - wp
    const df adw    = n1 ? dlt : neg(dlt); // |w - wp|
    const int nlep = P.eta0 > 30. ? 1 : 2; // e+ terms below 1e-13 of e- for eta_e > 30
#pragma unroll 1
    for (int e = 0; e < nlep; ++e)
    {
        const double eta = e ? P.eta1 : P.eta0;
        if (y > eta * 1e-3)
        {
            const df aw = from_double(eta - w), awp = from_double(eta - wp);
            const df aab = from_double(eta - ad);
            df rwp[5], rab[5];
            fdi_raw15(awp, rwp, 1, ftab);
            fdi_raw15(aab, rab, 3, ftab);
            rab[0] = rab[1] = Q.reta[e][0];
            df dw[5], d5[5];
            fdi_diff15(rw[e], rwp, aw, awp, dlt, dw);
            fdi_diff15(rab, Q.reta[e], aab, Q.eta[e], adw, d5);
            const df dabs[3] = {d5[2], d5[3], d5[4]};
            const df T1 = add(dw[3], mul(add(mul(S, dw[2]), mul(mul(Pp, 3.f), dw[1])), 2.f));
            const df U  = add(mul(X, dabs[1]), mul(mul(mul(X, X), 2.f), dabs[0]));
            const df V  = add(neg(mul(Y, dabs[1])), mul(mul(mul(Y, Y), 2.f), dabs[0]));
            constexpr dfc kFifth(0.2);
            const df c1 = sub(mul(mul(dabs[2], mk(kFifth)), sign1), mul(dw[4], mk(kFifth)));
            const df A1 = sub(div(add(sub(c1, mul(S, T1)), mul(U, sign1)), Dn), mul(dw[0], 6.f));
            const df B1 = div(add(c1, mul(V, sign1)), Dn);
            constexpr dfc kBp(k::NepsBPlus), kBm(k::NepsBMinus), kBz(k::NepsBZero);
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                const df bo      = (s < 2) ? mk(kBp) : mk(kBm);
                const bool first = ((s & 1) == 0) != (e == 1);
                const df r = first ? add(mul(A1, bo), mul(B1, mk(kBz)))
                                   : add(mul(A1, mk(kBz)), mul(B1, bo));
                R[s] += r.hi;
            }
        }
        else
        {
            double t1[4], t2[4];
            neps_taylor(P, e, w, wp, x, y, (int)sign1, n1 ? -1 : 1, t1, t2);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                R[s] += (float)t1[s];
        }
    }
}

} // namespace
} // namespace bnsn

namespace bnsn {
namespace {

// ---------------------------------------------------------------------------
// Spectral NES/NPS in FP32 with exponent scaling.
//
// At a fixed energy w = nu/T the NES emissivity integrand carries
// e^{-(w - w')} g(w') (w' < w) and the absorption integrand e^{-(w' - w)}
// (1 - g(w')) (w' > w): for w of tens to hundreds both leave the FP32 range
// while the integral itself is an ordinary FP64 number.  The occupation
// factors are therefore formed as exponentials of double-float arguments
// minus a per-energy shift sigma (an upper estimate of the largest log
// factor over the nodes), the terms are summed in those scaled units, and
// e^{sigma} is applied in FP64.  Components whose scaled value falls below
// 2^-120 are dropped and their bound is returned, so that the caller can
// recompute in FP64 when dropped or denormal terms could matter.
// ---------------------------------------------------------------------------
constexpr float kNesDrop    = 7.52316385e-37f; // 2^-120
constexpr float kNesDropArg = -83.1777f;       // log 2^-120

struct alignas(8) NesSpec
{
    dfm::df invTt[4], etat[4], invTf[4], cf[4], lbf[4], lwt[4], lwf[4];
    int has_t;  // bit s: w_t of species s nonzero
    int has_fe; // bit s: free part of species s nonzero (w_f > 0, beta_f > 0)
    int has_fa; // bit s: w_f of species s nonzero (enters 1 - g)
};

// Species data of one point (call for s = 0..3; the masks come from nes_spec_masks).
__device__ __forceinline__ void nes_spec_species(const Distr& d, int s, NesSpec* Z)
{
    Z->invTt[s] = dfm::from_double(1. / d.temp_t[s]);
    Z->etat[s]  = dfm::from_double(d.eta_t[s]);
    Z->invTf[s] = dfm::from_double(1. / d.temp_f[s]);
    Z->cf[s]    = dfm::from_double(d.c_f[s]);
    Z->lbf[s]   = dfm::from_double(d.beta_f[s] > 0. ? log(d.beta_f[s]) : 0.);
    Z->lwt[s]   = dfm::from_double(d.w_t[s] > 0. ? log(d.w_t[s]) : 0.);
    Z->lwf[s]   = dfm::from_double(d.w_f[s] > 0. ? log(d.w_f[s]) : 0.);
}

__device__ __forceinline__ void nes_spec_masks(const Distr& d, NesSpec* Z)
{
    int mt = 0, mfe = 0, mfa = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        mt |= (d.w_t[s] > 0.) << s;
        mfe |= (d.w_f[s] > 0. && d.beta_f[s] > 0.) << s;
        mfa |= (d.w_f[s] > 0.) << s;
    }
    Z->has_t  = mt;
    Z->has_fe = mfe;
    Z->has_fa = mfa;
}

// Largest estimated log occupation factor over nodes a0, a0 + step, ... < 2n
// of energy nu (w = nu/T): sig[0] for emission (g e^{-(w - w')^+}), sig[1]
// for absorption ((1 - g) e^{-(w' - w)^+}); -inf when there are no nodes.
// FP32 throughout: sigma is only a scale, its error cancels exactly.
__device__ __forceinline__ void nes_spec_scan(const NesSpec& Z, float w, float nu, float lnu,
                                              const double* x, const dfm::df* lx, int n, int a0,
                                              int step, bool nbb, float* sig)
{
    float se = -INFINITY, sa = -INFINITY;
    for (int a = a0; a < 2 * n; a += step)
    {
        const bool first = a < n;
        const int i      = first ? a : a - n;
        const float xi = (float)x[i], li = lx[i].hi;
        const float wp  = first ? w * xi : w / xi;
        const float nub = first ? nu * xi : nu / xi;
        const float lnb = first ? lnu + li : lnu - li;
        const float D   = fabsf(w - wp);
#pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            const bool ht = (Z.has_t >> s) & 1, hfe = (Z.has_fe >> s) & 1;
            const bool hfa = (Z.has_fa >> s) & 1;
            const float A  = nub * Z.invTt[s].hi - Z.etat[s].hi;
            const float Fn = Z.lbf[s].hi + Z.cf[s].hi * lnb - nub * Z.invTf[s].hi;
            const float le = fmaxf(ht ? Z.lwt[s].hi - fmaxf(A, 0.f) : -INFINITY,
                                   hfe ? Z.lwf[s].hi + Fn : -INFINITY);
            const float la = nbb ? 0.f
                                 : fmaxf(ht ? Z.lwt[s].hi - fmaxf(-A, 0.f) : -INFINITY,
                                         hfa ? Z.lwf[s].hi : -INFINITY);
            se = fmaxf(se, first ? le - D : le);
            sa = fmaxf(sa, first ? la : la - D);
        }
    }
    sig[0] = se;
    sig[1] = sa;
}

// exp of a double-float argument in FP32 (first-order remainder factor).
__device__ __forceinline__ float exp_of(dfm::df x) { return expf(x.hi) * (1.f + x.lo); }

// NES/NPS terms of one spectral node for the four species, in scaled units:
//   te[s] = wa w'^2 R_s (+-E/dn) g_s e^{-sig_e},
//   ta[s] = wa w'^2 R_s (+-E/dn) (1 - g_s) e^{-sig_a},
// where E = e^{-|w - w'|} sits in the emission factor for w' < w and in the
// absorption factor for w' > w, and dn = 1 - E (NEPSExpFunc,
// functions.hpp:4401-4413).  de[s], da[s] bound the dropped components of
// te[s], ta[s].
// Node arguments in df: W = nu/T, WP = nubar/T, NB = nubar, LB = log nubar
// (w, wp the same in FP64 for the kernel).  fw: the Fermi integrals at eta_e - w,
// phi_1..phi_5, or with Q (double-float kernel) the unreflected F_1..F_5 in df.
__device__ __forceinline__ void nes_spec_node(const NepsPoint& P, const NesSpec& Z, double w,
                                              double wp, dfm::df W, dfm::df WP, dfm::df NB,
                                              dfm::df LB, float wa, float sig_e, float sig_a,
                                              bool nbb, const double (*fw)[5], const NesDf* Q,
                                              const dfm::FdiTab* ftab, float* te, float* ta,
                                              float* de, float* da)
{
    using namespace dfm;
    float R[4];
    if (Q) // known at compile time
        neps_r_df(P, *Q, ftab, w, wp, W, WP, (const dfm::df (*)[5])fw, R);
    else
        neps_r_mixed(P, w, wp, fw, R);
    const bool first = wp < w;
    const df D       = first ? sub(W, WP) : sub(WP, W); // |w - wp|
    const float ea   = expf(-D.hi);
    const float dn   = -expm1f(-D.hi) + ea * D.lo; // 1 - e^{-D}
    const df Se = first ? add(D, sig_e) : mk(sig_e);
    const df Sa = first ? mk(sig_a) : add(D, sig_a);
    const float c = (first ? wa : -wa) * (WP.hi * WP.hi) / dn;
    float gnb = 0.f, unb = 0.f; // neglected blocking: (1 - g) -> 1
    if (nbb)
    {
        const df x = neg(Sa);
        if (x.hi < kNesDropArg)
            unb = kNesDrop;
        else
            gnb = exp_of(x);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        const bool ht = (Z.has_t >> s) & 1, hfe = (Z.has_fe >> s) & 1;
        const bool hfa = (Z.has_fa >> s) & 1;
        float ge = 0.f, gm = nbb ? gnb : 0.f, le = 0.f, la = nbb ? unb : 0.f;
        if (ht)
        {
            const df A      = sub(mul(NB, Z.invTt[s]), Z.etat[s]);
            const float inv = 1.f / (1.f + expf(-fabsf(A.hi)));
            const bool pos  = A.hi > 0.f;
            const df x1     = sub(pos ? sub(Z.lwt[s], A) : Z.lwt[s], Se);
            if (x1.hi < kNesDropArg)
                le += kNesDrop;
            else
                ge += exp_of(x1) * inv;
            if (!nbb)
            {
                const df x3 = sub(pos ? Z.lwt[s] : add(Z.lwt[s], A), Sa);
                if (x3.hi < kNesDropArg)
                    la += kNesDrop;
                else
                    gm += exp_of(x3) * inv;
            }
        }
        df Fn = mk(0.f);
        if (hfe)
        {
            Fn          = add(Z.lbf[s], sub(mul(Z.cf[s], LB), mul(NB, Z.invTf[s])));
            const df x2 = add(Fn, sub(Z.lwf[s], Se));
            if (x2.hi < kNesDropArg)
                le += kNesDrop;
            else
                ge += exp_of(x2);
        }
        if (hfa && !nbb)
        {
            const df x4 = sub(Z.lwf[s], Sa);
            // 1 - f_free = -expm1(log f_free), accurate when f_free is near 1
            const float omf = hfe ? -(expm1f(Fn.hi) + expf(Fn.hi) * Fn.lo) : 1.f;
            if (x4.hi < kNesDropArg)
                la += kNesDrop;
            else
                gm += exp_of(x4) * omf;
        }
        const float k = c * R[s];
        te[s] = k * ge;
        ta[s] = k * gm;
        de[s] = fabsf(k) * le;
        da[s] = fabsf(k) * la;
    }
}

} // namespace
} // namespace bnsn
