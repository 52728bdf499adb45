// Grey M1 opacity kernels (sm_103a), FP64 and mixed precision.
//
// Restates ComputeM1OpacitiesGenericFormalism (m1_opacities.hpp:1062-1295)
// with the integration rules of integration.hpp:608-844, as six phase
// kernels over a chunk of points.  Each phase has a small hot loop shared by
// all resident warps, so the instruction working set stays in the SM's
// instruction cache (a single fused kernel spent most of its issue slots
// waiting on instruction fetch):
//
//   point   : per (point, task) (one thread): distribution parameters,
//             Fermi integrals at +-eta_e, brem, beta and iso constants, written to
//             the header of the point's scratch record.
//   prelude : per point (four warps): the 2n-energy tables of the double
//             integral (distribution values, F_k(eta +- w/T)) and the 1-D beta
//             and iso-scattering integrals.
//   pair    : per point (64 threads): the M(M+1)/2 unordered (w, w') cells of the
//             pair kernel, one evaluation filling (w, w') and (w', w) of a kernel
//             matrix in shared memory, then its rows weighted and summed into the
//             number and energy moments.
//   brem    : the same for the bremsstrahlung kernel (HR98, BRT06, GP19).
//   neps    : per point (two warps): the 2 n^2 (nu, nubar) pairs of the NES/NPS
//             double integral, both directions from one set of Fermi integrals.
//   final   : per (point, species) (one thread): assembly of the 20 outputs.
//
// Calls of few points take a point per wider CTA in pair, brem and neps, and run the
// three in one launch; a point's results do not depend on the form.
//
// FP64 path: every sum and weight in FP64; exponentials, logarithms, powers and the Fermi
// integrals in 64-bit fixed point on the integer pipes (bnsn_fx.cuh), to an ulp.
// Mixed path: FP32 pair (bnsn_pair32.cuh), NES (bnsn_nes32.cuh) and brem kernels
// (bnsn_fp32.cuh) and occupations with double-float exponent arguments; the weights
// and sums stay FP64 (brem and NES terms are summed in FP32 and double-float runs), and
// sums that cancel are recomputed in FP64.

#include <cuda_runtime.h>

#include "bnsn_df.cuh"
#include "bnsn_fp32.cuh"
#include "bnsn_mixed.cuh"
#include "bnsn_fp64.cuh"
#include "bnsn_nes32.cuh"
#include "bnsn_pair32.cuh"
#include "bnsn_internal.h"

namespace bnsn {

using namespace fp64;

// Per-point record in the scratch arena (double words only, no padding).
struct PointTab
{
    Distr d;
    double fe[2][6];  // F_0..F_5 at eta_e and -eta_e
    double fd0[2];    // FermiDistr(0, 1, +-eta_e)
    Hr98Point hr;
    double brt06_pre;
    double eta_pp, eta_nn;
    double spare;
    double nu[kMaxM];    // energies of the double-integral grid
    double y[kMaxM];     // nu / T
    double g[kMaxM][4];  // TotalNuF at nu per species
    double fm[kMaxM][5]; // F_1..F_5 at eta_e - nu/T
    double fp[kMaxM][5]; // F_1..F_5 at eta_e + nu/T
    double s2d[16];      // pair + brem: n-moment em/ab, J-moment em/ab
    double snes[16];     // NES/NPS, same layout
    double sbeta[8];     // beta: n_em[2], j_em[2], n_ab[2], j_ab[2]
    double siso[4];      // iso per species
    double sbrem[16];    // brem alone (its part of s2d)
    double bmag[16];     // mixed path: sum of |term| of FP32 brem cells (s2d units), else 0
    double neps_fp64;    // mixed path: not 0 if the NES sums of the point must be FP64
    double bredo;        // mixed path: 1 if the brem sums must be recomputed in FP64
};
static_assert(sizeof(PointTab) % sizeof(double) == 0, "PointTab must be double words");
static_assert(sizeof(PointTab) == kGreyRecordBytes, "grey record size");
constexpr int kTabWords = sizeof(PointTab) / sizeof(double);

// Mixed path with the pair kernel on: the pair phase computes no Fermi-integral
// tables (fm, fp), so their words hold its own sums, their magnitudes and the
// final kernel's verdict instead.
struct PairMixed
{
    double spair[16]; // the pair part of s2d
    double pmag[16];  // sum of |term| of the pair cells per moment (s2d units)
    double predo;     // 1 if the point's pair sums must be recomputed in FP64
};
static_assert(sizeof(PairMixed) <= sizeof(((PointTab*)nullptr)->fm), "PairMixed overlay");
// Mixed path: points evaluated, points whose FP32 NES sums cancel and those outside
// the FP32 range (NES in FP64), pair sums redone in FP64, brem sums redone in FP64 (read by
// grey_mixed_counts).
__device__ unsigned long long g_grey_mixed[5];

__device__ __forceinline__ PairMixed* pair_mixed(PointTab* P)
{
    return reinterpret_cast<PairMixed*>(&P->fm[0][0]);
}

// GP19 brem: the point's extrapolation regime and the corners of its profiles
// take the words of the HR98 constants.
struct Gp19Record
{
    Gp19Point pt;
    Gp19Corners cor[2];
};
static_assert(sizeof(Gp19Record) <= sizeof(Hr98Point), "Gp19Record overlay");

__device__ __forceinline__ Gp19Record* gp19_record(PointTab* P)
{
    return reinterpret_cast<Gp19Record*>(&P->hr);
}

size_t grey_point_scratch_bytes() { return sizeof(PointTab); }

namespace {

constexpr int kWarps = 4; // warps per CTA in the per-point kernels

// Sums the 16 values of the warp's lanes: lane l returns the total of value
// sum_index(l).  Each round halves the values a lane carries, 16 additions in
// all instead of 80 for 16 butterfly sums.
__device__ __forceinline__ double warp_sum16(double* v, int lane)
{
#pragma unroll
    for (int n = 8, o = 16; n >= 1; n >>= 1, o >>= 1)
    {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < n; ++k)
        {
            const double mine = up ? v[k + n] : v[k], theirs = up ? v[k] : v[k + n];
            v[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}
__device__ __forceinline__ int sum_index(int lane)
{
    return ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
}

// Cooperative copy of `words` doubles (lane-strided, coalesced).
__device__ __forceinline__ void warp_copy(double* __restrict__ dst,
                                          const double* __restrict__ src, int words,
                                          int lane)
{
    for (int k = lane; k < words; k += 32)
        dst[k] = src[k];
}

// s_beta of m1_opacities.hpp:1093-1110 of species s (0, 1) from F_4, F_5 at +-eta_e.
__device__ __forceinline__ double beta_scale(double f4, double f5, double T, double eta_e, int s)
{
    if (eta_e > -30. && eta_e < 30.)
        return T * f5 / f4;
    return (eta_e > 30.) == (s == 0) ? T * eta_e * 0.8333333333333333 : T * 5.;
}

// TotalNuF of one species in FP32 with its exponent arguments in df form
// (distribution.hpp:298-315): x rt - eta_t and P0 + c_f log x - x rf.  The
// NES items take x = w = omega / T (rt = T / T_t, rf = T / T_f,
// P0 = log beta_f + c_f log T), the prelude's beta and iso items x = omega
// in MeV (rt = 1 / T_t, rf = 1 / T_f, P0 = log beta_f).  Both arguments cancel
// (the product's leading part against eta_t or P0), so they are formed from
// the exact FMA remainders; the occupation and its complement then keep FP32
// relative accuracy (the complement from the two parts' complements,
// w_t + w_f = 1 for the reconstructed distribution).
struct NuSpecies
{
    dfm::df etat, rt, P0, cf, rf;
    float wt, wf;
};

__device__ __forceinline__ void total_nu_one(dfm::df X, dfm::df LX, const NuSpecies& S,
                                             float& g, float& gm)
{
    // a = x rt - eta_t as hi + lo; e^{-|a|} = e^{-|hi|} (1 -+ lo): a float
    // exponent alone would cost |a| 6e-8 of relative accuracy
    const dfm::df pa = dfm::two_prod(X.hi, S.rt.hi);
    const dfm::df sa = dfm::two_sum(pa.hi, -S.etat.hi);
    const dfm::df A  = dfm::fast_two_sum(
        sa.hi, sa.lo + pa.lo + fmaf(X.hi, S.rt.lo, fmaf(X.lo, S.rt.hi, -S.etat.lo)));
    const bool pos  = A.hi > 0.f;
    const float t   = expf(-fabsf(A.hi)) * (pos ? 1.f - A.lo : 1.f + A.lo);
    const float inv = nes32::rcp_nr(t + 1.f);
    const float ft  = pos ? t * inv : inv;
    const float ftm = pos ? inv : t * inv;
    float fn        = 0.f;
    if (S.wf != 0.f)
    {
        const dfm::df p1 = dfm::two_prod(S.cf.hi, LX.hi);
        const dfm::df p2 = dfm::two_prod(-X.hi, S.rf.hi);
        const dfm::df s1 = dfm::two_sum(S.P0.hi, p1.hi);
        const dfm::df s2 = dfm::two_sum(s1.hi, p2.hi);
        const float lo   = (S.P0.lo + p1.lo + p2.lo + s1.lo + s2.lo) +
                         fmaf(S.cf.hi, LX.lo, S.cf.lo * LX.hi) - fmaf(X.hi, S.rf.lo, X.lo * S.rf.hi);
        const dfm::df F = dfm::fast_two_sum(s2.hi, lo);
        fn = expf(F.hi) * (1.f + F.lo);
    }
    g  = S.wt * ft + S.wf * fn;
    gm = S.wt * ftm + S.wf * (1.f - fn);
}

// The constants of species s of distribution d for x = omega * xscale
// (xscale = 1 / T for the NES items, 1 for omega in MeV); lxs = log xscale.
__device__ __forceinline__ void nu_species(const Distr& d, int s, double xscale_inv, double lxs,
                                           NuSpecies* S)
{
    S->wt   = (float)d.w_t[s];
    S->wf   = (float)d.w_f[s];
    S->etat = dfm::from_double(d.eta_t[s]);
    S->rt   = dfm::from_double(xscale_inv / d.temp_t[s]);
    const double lbf = d.beta_f[s] > 0. ? fx::log(d.beta_f[s]) : 0.;
    S->P0   = dfm::from_double(lbf - d.c_f[s] * lxs);
    S->cf   = dfm::from_double(d.c_f[s]);
    S->rf   = dfm::from_double(xscale_inv / d.temp_f[s]);
}

// The four species; with nocc = 3 species 3 equals species 2.
__device__ __forceinline__ void total_nu_q(dfm::df W, dfm::df LW, const NuSpecies* sp, int nocc,
                                           float* g, float* gm)
{
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        if (s < nocc)
            total_nu_one(W, LW, sp[s], g[s], gm[s]);
        else
        {
            g[s]  = g[2];
            gm[s] = gm[2];
        }
    }
}

// What the prelude needs beyond the record's header, written by the point kernel
// into the words of the sums that later phases fill (s2d .. bmag).
struct PreRecord
{
    double rt[4], rf[4], kf[4]; // Occ64 of omega in MeV
    NuSpecies nu[4];            // mixed path
    BetaPoint bp;
    double t[6], lt[6];         // energy scales of beta (2) and iso (4), their logs (mixed)
};
static_assert(sizeof(PreRecord) <= 76 * sizeof(double), "PreRecord overlay (s2d .. bmag)");

__device__ __forceinline__ PreRecord* pre_record(PointTab* P)
{
    return reinterpret_cast<PreRecord*>(&P->s2d[0]);
}

// ---------------------------------------------------------------------------
// point constants: the per-point quantities that do not depend on an energy
// node, as 13 independent tasks, one thread per (point, task) with the task
// in blockIdx.y (every warp runs one code path):
//   0..3  distribution parameters of species 0..3 (or a copy of the given ones),
//         their occupation constants and the iso integral's energy scale
//   4, 5  F_0..F_5 and FermiDistr(0, 1, .) at +eta_e, -eta_e, the beta scale
//   6..8  HR98 channel constants; 9: HR98 point constants; 10: BRT06 prefactor
//   6, 7  GP19: the point's regime and the corners of its two profiles
//   11    eta_NN of protons and neutrons (iso scattering)
//   12    beta-process constants
// written straight into the point's scratch record, whose header the prelude
// then loads.  Inside the one-warp-per-point prelude these tasks ran on one to
// four lanes each, one after the other.
// ---------------------------------------------------------------------------
constexpr int kPointTasks = 13;

template <bool MULTI = false>
__global__ void __launch_bounds__(128)
    grey_point_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                      int64_t np, double* __restrict__ scratch)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    const int task = blockIdx.y;
    const bool gp19 = L.use_brem && L.brem_impl == 2 && L.gp19.d3 <= kGp19MaxW;
    if ((task >= 6 && task <= 9 && !(L.use_brem && L.brem_impl == 0) && !(gp19 && task < 8)) ||
        (task == 10 && !(L.use_brem && L.brem_impl == 1)) || (task == 11 && !L.use_iso) ||
        (task == 12 && !L.use_abs_em))
        return;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < np;
         q += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        const double nb = L.eos[0][p], T = L.eos[1][p];
        if (task < 4)
        {
            const int s = task;
            Distr& d    = P->d;
            if (L.has_distr)
            {
#pragma unroll
                for (int f = 0; f < 7; ++f)
                    (&d.w_t[0])[f * 4 + s] = L.distr[f * 4 + s][p];
            }
            else
                distr_species(L.m1[s][p], L.m1[4 + s][p], L.m1[8 + s][p], L.gamma36, &d.w_t[s],
                              &d.temp_t[s], &d.eta_t[s], &d.w_f[s], &d.temp_f[s], &d.c_f[s],
                              &d.beta_f[s]);
            PreRecord* R = pre_record(P);
            Occ64 o;
            occ64_from(d, s, 1., &o);
            R->rt[s] = o.rt;
            R->rf[s] = o.rf;
            R->kf[s] = o.kf;
            const double ns = L.m1[s][p];
            const double t  = (ns > k::ThresholdN) ? (L.m1[4 + s][p] / ns) : 1.5 * T;
            R->t[2 + s] = t;
            if (L.mixed)
            {
                nu_species(d, s, 1., 0., &R->nu[s]);
                R->lt[2 + s] = fx::log(t);
            }
        }
        else if (task < 6)
        {
            const int e     = task - 4;
            const double et = e ? -L.eos[7][p] / T : L.eos[7][p] / T;
            double f[6];
            fdi_orders<0, 5>(et, f);
#pragma unroll
            for (int kk = 0; kk < 6; ++kk)
                P->fe[e][kk] = f[kk];
            P->fd0[e]      = fermi_distr(0., 1., et);
            const double t = beta_scale(f[4], f[5], T, e ? -et : et, e);
            pre_record(P)->t[e] = t;
            if (L.mixed)
                pre_record(P)->lt[e] = fx::log(t);
        }
        else if (task < 9 && gp19)
        {
            const Gp19Table G = {L.gp19.d0, L.gp19.d1, L.gp19.d2, L.gp19.d3,
                                 L.gp19.nb, L.gp19.ye, L.gp19.t,  L.gp19.w,
                                 L.gp19.lognb, L.gp19.logw, L.gp19.data};
            Gp19Point pt;
            gp19_point(G, nb, L.eos[2][p], T, &pt);
            Gp19Record* R = gp19_record(P);
            if (task == 6)
                R->pt = pt;
            if (task == 6 || pt.regime >= 2)
                gp19_profile_corners(G, pt.nbp, pt.yep, pt.pT[task - 6], &R->cor[task - 6]);
        }
        else if (task < 9)
            P->hr.ch[task - 6] = hr98_channel(nb, L.eos[4][p], L.eos[3][p], T, task - 6);
        else if (task == 9)
            hr98_point_common(nb, T, L.use_medium != 0, &P->hr); // leaves hr.ch alone
        else if (task == 10)
            P->brt06_pre = brt06_point(nb, T, L.eos[4][p], L.eos[3][p]);
        else if (task == 12)
            pre_record(P)->bp = beta_point(nb, T, L.eos[3][p], L.eos[4][p], L.eos[5][p],
                                           L.eos[6][p], L.eos[7][p], L.eos[9][p], L.eos[10][p],
                                           L.use_dU, L.use_dm_eff, L.use_WM_ab, L.use_decay);
        else
        {
            P->eta_pp = eta_nn_sc(nb, T, L.eos[3][p]);
            P->eta_nn = eta_nn_sc(nb, T, L.eos[4][p]);
        }
    }
}

// ---------------------------------------------------------------------------
// prelude: the energy tables of the double integral (m1_opacities.hpp:783-787),
// the beta integrals (m1_opacities.hpp:93-237, integration.hpp:805-844) and the
// iso-energetic scattering integrals (m1_opacities.hpp:39-91, integration.hpp:
// 770-802).  Four warps share a point; a warp takes every fourth of the point's
// units of 32 nodes of one kind (2 units of occupations, 3 of Fermi integrals, 3
// of beta and 5 of iso nodes at n = 20), so that warps do not diverge and a
// single point's chain is four units long.  FP64 pipe bound.  8,192 points, n =
// 20: 1.09 -> 0.68 ms, mixed 0.81 -> 0.44 ms; one point, n = 10: 94 -> 46 us
// (with the point kernel).
// ---------------------------------------------------------------------------
constexpr int kPreWarps = 4;

struct PreSmem
{
    double B1[kMaxM], x1[kMaxM];       // 1-D nodes x_i and 1 / x_i, their weights
    double y2[kMaxM], lx1[kMaxM];      // 2-D nodes nu / T, log of the 1-D nodes
    double red[kPreWarps][12];
    Occ64 occ[4];
    PreRecord R;
};

template <bool MULTI = false>
__global__ void __launch_bounds__(kPreWarps * 32, 4)
    grey_prelude_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                        int64_t np, double* __restrict__ scratch)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    __shared__ PreSmem S;
    const int n1 = L.n1, n2 = L.n2, M = 2 * n2, M1 = 2 * n1;
    for (int k = threadIdx.x; k < kMaxM; k += blockDim.x)
    {
        S.B1[k] = L.B1[k];
        if (k < M1)
        {
            const int i = k < n1 ? k : k - n1;
            S.x1[k]     = k < n1 ? L.x1[i] : 1. / L.x1[i];
            S.lx1[k]    = k < n1 ? L.lx1[i] : -L.lx1[i];
        }
        if (k < M)
            S.y2[k] = k < n2 ? k::TempMultiple * L.x2[k] : k::TempMultiple / L.x2[k - n2];
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool mixed = L.mixed != 0;
    // units of each kind
    const int u_node = (L.use_pair || L.use_brem) ? (M + 31) / 32 : 0;
    const int u_fdi  = u_node + (L.use_pair && !mixed ? (2 * M + 31) / 32 : 0);
    const int u_beta = u_fdi + (L.use_abs_em ? (2 * M1 + 31) / 32 : 0);
    const int u_iso  = u_beta + (L.use_iso ? (4 * M1 + 31) / 32 : 0);

    for (int64_t q = blockIdx.x; q < np; q += gridDim.x)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        const double T = L.eos[1][p], eta_e = L.eos[7][p] / T;
        __syncthreads(); // the previous point's readers are done
        for (int k = threadIdx.x; k < (int)(sizeof(PreRecord) / sizeof(double)); k += blockDim.x)
            ((double*)&S.R)[k] = ((const double*)pre_record(P))[k];
        if (threadIdx.x >= 96 && threadIdx.x < 100)
        {
            const int s  = threadIdx.x - 96;
            S.occ[s].eta = occ64_eta(P->d, s);
            S.occ[s].wt  = P->d.w_t[s];
            S.occ[s].cf  = P->d.c_f[s];
        }
        __syncthreads();
        if (threadIdx.x < 4)
        {
            const int s = threadIdx.x;
            S.occ[s].rt = S.R.rt[s];
            S.occ[s].rf = S.R.rf[s];
            S.occ[s].kf = S.R.kf[s];
        }
        __syncthreads();
        const double c0    = S.occ[0].cf;
        const bool same_cf = S.occ[1].cf == c0 && S.occ[2].cf == c0 && S.occ[3].cf == c0;
        const double eta_pp = P->eta_pp, eta_nn = P->eta_nn;
        // a lane's species is fixed: lane & 1 in the beta units, lane & 3 in the iso units
        double bn_em = 0., bj_em = 0., bn_ab = 0., bj_ab = 0., iso_sum = 0.;
#pragma unroll 1
        for (int u = wid; u < u_iso; u += kPreWarps)
        {
            if (u < u_node)
            {
                const int a = u * 32 + lane;
                if (a < M)
                {
                    const double y = S.y2[a], nu = y * T;
                    double g[4];
                    occ64_eval(S.occ, nu, same_cf ? fx::pow(nu, c0) : 0., same_cf, g);
                    P->nu[a] = nu;
                    P->y[a]  = y;
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        P->g[a][s] = g[s];
                }
            }
            else if (u < u_fdi)
            {
                const int t = (u - u_node) * 32 + lane;
                if (t < 2 * M)
                {
                    const double y = S.y2[t >> 1];
                    double f[5];
                    fdi_orders<1, 5>(t & 1 ? eta_e + y : eta_e - y, f);
                    double* o = t & 1 ? P->fp[t >> 1] : P->fm[t >> 1];
#pragma unroll
                    for (int k = 0; k < 5; ++k)
                        o[k] = f[k];
                }
            }
            else
            {
                const bool beta = u < u_beta;
                const int it    = (u - (beta ? u_fdi : u_beta)) * 32 + lane;
                const int s     = it & (beta ? 1 : 3), a = it >> (beta ? 1 : 2);
                if (a < M1)
                {
                    const int sc    = beta ? s : 2 + s;
                    const double nu = S.R.t[sc] * S.x1[a];
                    double g;
                    if (mixed)
                    {
                        float gf, gmf;
                        total_nu_one(dfm::from_double(nu), dfm::from_double(S.R.lt[sc] + S.lx1[a]),
                                     S.R.nu[s], gf, gmf);
                        g = gf;
                    }
                    else
                        g = occ64_one(S.occ[s], nu, fx::pow(nu, S.occ[s].cf));
                    const double nu2 = nu * nu, w2 = S.B1[a] * nu2;
                    if (beta)
                    {
                        double ab, em;
                        beta_rates(S.R.bp, nu, s, &ab, &em);
                        if (L.stim)
                            ab = ab + em;
                        const double ev = w2 * em, av = w2 * (g * ab);
                        bn_em += ev;
                        bn_ab += av;
                        bj_em = fma(nu, ev, bj_em);
                        bj_ab = fma(nu, av, bj_ab);
                    }
                    else
                    {
                        // mixed: the weak-magnetism factors in FP32 (positive terms; the
                        // iso sum enters kappa_s alone, no other reaction cancels it)
                        const double iso =
                            (mixed && L.use_WM_sc)
                                ? k::IsoConst *
                                      (eta_pp * (double)fp32::iso_wm_factor((float)nu, 1) +
                                       eta_nn * (double)fp32::iso_wm_factor((float)nu, 2))
                                : iso_scatt_total(nu, eta_pp, eta_nn, L.use_WM_sc != 0);
                        iso_sum = fma(4. * k::Pi * (nu2 * nu) * w2, g * iso, iso_sum);
                    }
                }
            }
        }
        // lanes of one species; then the four warps
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1)
            iso_sum += __shfl_xor_sync(0xffffffffu, iso_sum, o);
        {
            const bool hi = (lane & 16) != 0, hj = (lane & 8) != 0;
            const double a0 = (hi ? bn_ab : bn_em) +
                              __shfl_xor_sync(0xffffffffu, hi ? bn_em : bn_ab, 16);
            const double a1 = (hi ? bj_ab : bj_em) +
                              __shfl_xor_sync(0xffffffffu, hi ? bj_em : bj_ab, 16);
            double b = (hj ? a1 : a0) + __shfl_xor_sync(0xffffffffu, hj ? a0 : a1, 8);
            b += __shfl_xor_sync(0xffffffffu, b, 4);
            b += __shfl_xor_sync(0xffffffffu, b, 2);
            // sbeta order: n_em, j_em, n_ab, j_ab of species 0, 1
            if ((lane & 6) == 0)
                S.red[wid][(hi ? 4 : 0) + (hj ? 2 : 0) + (lane & 1)] = b;
            if (lane < 4)
                S.red[wid][8 + lane] = iso_sum;
        }
        __syncthreads();
        if (threadIdx.x < 12)
        {
            const int k = threadIdx.x;
            double t    = S.red[0][k];
#pragma unroll
            for (int w = 1; w < kPreWarps; ++w)
                t += S.red[w][k];
            if (k < 8)
                P->sbeta[k] = t;
            else
                P->siso[k - 8] = t;
        }
    }
}

// Shared-memory copy of the energy tables the FP32 brem cells need.
struct CellTab
{
    double nu[kMaxM];
    double y[kMaxM];
    double g[kMaxM][4];
    double brt06_pre;
    fp32::Hr98Mixed hm;
};

__device__ __forceinline__ void load_cell_tab(CellTab& C, const PointTab* __restrict__ P,
                                              int M, int lane)
{
    warp_copy(C.nu, P->nu, M, lane);
    warp_copy(C.y, P->y, M, lane);
    warp_copy(&C.g[0][0], &P->g[0][0], 4 * M, lane);
    if (lane == 0)
        C.brt06_pre = P->brt06_pre;
}

// Mixed-path cell tables (FP32): g and 1 - g per species (1 - g formed in
// FP64), and nu/T as a double-float pair for the detailed-balance exponent.
struct CellTab32
{
    float g[kMaxM][4];
    float gm[kMaxM][4];
    float yh[kMaxM], yl[kMaxM];
};

// FP32 cell sums: per-lane partial sums of up to 4 cells are flushed into the
// FP64 accumulators, which bounds the FP32 summation error by a few ulp.
struct Acc32
{
    float v[16];
    float mag[16]; // sum of |term| per moment
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int k = 0; k < 16; ++k)
            v[k] = 0.f;
    }
};

// The beta rate of element idx of a point's 16 sums in the units of the pair/brem
// sums (s2d, unit t2 = (2.182 T)^2 for number and t2d t2 for energy moments) or, with
// to_nes, of the NES sums (unit hn = 8 t2, times T for energy moments), as
// the final assembly combines them (m1_opacities.hpp:1172-1294).
__device__ __forceinline__ double beta_in_sum_unit(const PointTab* P, double T, double eta_e,
                                                   bool use_abs_em, bool to_nes, int idx)
{
    const int s = idx & 3, m = idx >> 2; // species; number em, ab, energy em, ab
    if (!use_abs_em || s >= 2)
        return 0.;
    const double sb = beta_scale(P->fe[s][4], P->fe[s][5], T, eta_e, s);
    const double t2d = k::TempMultiple * T, t2 = t2d * t2d;
    const double un  = k::FourPiHc3 * (to_nes ? 8. * t2 : t2);
    const double u   = (m >= 2 && !to_nes) ? un * t2d : un;
    return P->sbeta[(m & 1) * 4 + (m >> 1) * 2 + s] * sb / u;
}

// Mixed sums whose terms cancel by more than this are recomputed in FP64: the
// FP32 rounding of each term (a few 1e-7) must stay below 1e-6 in the result.
constexpr double kMaxCancel = 2.0;
// FP32 brem cells carry up to ~6e-7 per term (the HR98 fit in FP32).
constexpr double kMaxCancelBrem = 1.25;
// FP32 pair integrals carry up to ~3e-7 per cell.
constexpr double kMaxCancelPair = 1.5;

// add_cell in FP32 for a species-independent kernel (brem): K_em, K_ab are
// dimensionless; P1 = (y_a y_b)^2 W1 and P2 = (y_a y_b)^2 W2 are the cell's
// weights with the energy factor, each one FP32 rounding of a double-float
// product (cell_weight); the caller scales by T^4 and the kernel's prefactor.
template <bool STIM>
__device__ __forceinline__ void add_cell32(Acc32& A, float Kem, float Kab, const float* ga,
                                           const float* gma, const float* gb, const float* gmb,
                                           bool nb_block, float P1, float P2)
{
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        const int ps   = s ^ 1;
        const float em = Kem * (nb_block ? 1.f : gmb[ps]);
        const float am = Kab * gb[ps];
        float EM, AB;
        if (STIM)
        {
            AB = ga[s] * (em + am);
            EM = em;
        }
        else
        {
            AB = am * ga[s];
            EM = em * gma[s];
        }
        const float e1 = EM * P1, a1 = AB * P1;
        A.v[s] += e1;
        A.v[4 + s] += a1;
        const float e2 = EM * P2, a2 = AB * P2;
        A.v[8 + s] += e2;
        A.v[12 + s] += a2;
        A.mag[s] += fabsf(e1);
        A.mag[4 + s] += fabsf(a1);
        A.mag[8 + s] += fabsf(e2);
        A.mag[12 + s] += fabsf(a2);
    }
}

// (y_a y_b)^2 w_a w_b rounded once to FP32 from double-float factors (in
// FP32 the fourth power alone magnified the rounding of y to 3e-7).
__device__ __forceinline__ float cell_weight(dfm::df w4, dfm::df wa, dfm::df wb)
{
    const dfm::df p = dfm::mul(w4, dfm::mul(wa, wb));
    return p.hi + p.lo;
}

// FP32 tables of one point from the FP64 ones.
__device__ __forceinline__ void fill_tab32(CellTab32& D, const CellTab& C, int M, int lane)
{
    for (int e = lane; e < 4 * M; e += 32)
    {
        const double gv     = C.g[e >> 2][e & 3];
        D.g[e >> 2][e & 3]  = (float)gv;
        D.gm[e >> 2][e & 3] = (float)(1. - gv);
    }
    for (int a = lane; a < M; a += 32)
    {
        const dfm::df yd = dfm::from_double(C.y[a]);
        D.yh[a]          = yd.hi;
        D.yl[a]          = yd.lo;
    }
}

// ---------------------------------------------------------------------------
// Cell phases with row sums.  A symmetric pair of cells (a, b), (b, a) costs one
// kernel evaluation; its weighting into the 16 moments of m1_opacities.hpp:577-758
// took ~100 FP64 operations per pair, more than the kernel itself.  The moments
// are bilinear in node vectors, so the phase first stores the absorption kernel
// K(a, b) of all cells in shared memory and then sums rows:
//   F_a = dn_a sum_b K(a, b) dn_b q_b (1 - g_b)   (emission: K e^{-(y_a + y_b)}),
//   G_a = sum_b K(a, b) q_b g_b,
// per partner species, after which a row adds q_a F_a, q_a g_a (F_a + G_a) and
// the same with the energy weight: 8 operations per directed cell (16 where
// K(b, a) != K(a, b)) and ~45 per row.  Two warps share a point (64 threads: 13
// and 4 rounds of cells at n = 20 and 10, 12 to 25 KB of shared memory per
// point).
// ---------------------------------------------------------------------------
constexpr int kCellThreads = 64, kCellWide = 256;

template <int NT>
struct CellNodes
{
    double K[kMaxM][kMaxM + 1];        // absorption kernel of (row, column)
    double vE[kMaxM][4], vA[kMaxM][4]; // q dn (1 - g), q g
    double g[kMaxM][4];
    double q[kMaxM], qe[kMaxM]; // number and energy weights of a node
    double dn[kMaxM];           // e^{-y}
    double nu[kMaxM], y[kMaxM];
    double red[2][NT / 32][16];
    double A1[kMaxM], A2[kMaxM];
    uint16_t cells[kMaxCells]; // a | b << 8
    int splits;                // column ranges a row is cut into
};

// Launch constants of the CTA, and the column split: rows x splits tasks of
// (M / splits) columns over the CTA's threads, chosen for the fewest rounds x
// (columns x products + the row's epilogue).
template <bool SYM, int NT>
__device__ __forceinline__ void cell_constants(CellNodes<NT>& C, const OpacityLaunch& L)
{
    const int M = 2 * L.n2;
    for (int k = threadIdx.x; k < kMaxM; k += NT)
    {
        C.A1[k] = L.A1[k];
        C.A2[k] = L.A2[k];
    }
    for (int k = threadIdx.x; k < L.ncell; k += NT)
    {
        const uint32_t ab = L.cells[k];
        C.cells[k]        = (uint16_t)((ab & 0xffu) | ((ab >> 16) << 8));
    }
    if (threadIdx.x == 0)
    {
        int best = 1, cost = 1 << 30;
        for (int h = 1; h <= 8 && h <= M; ++h)
        {
            const int c = ((M * h + NT - 1) / NT) *
                          (((M + h - 1) / h) * (SYM ? 8 : 16) + 45);
            if (c < cost)
            {
                cost = c;
                best = h;
            }
        }
        C.splits = best;
    }
}

// Node data of a point; nu2: the weights carry nu^2 (kernels without it).
template <int NT>
__device__ __forceinline__ bool cell_nodes(CellNodes<NT>& C, const PointTab* __restrict__ P, int M,
                                           bool nbb, bool nu2)
{
    bool above = false; // an occupation above 1
    const int a = threadIdx.x;
    if (a < M)
    {
        const double nu = P->nu[a], y = P->y[a];
        const double w  = nu2 ? nu * nu : 1.;
        const double q  = C.A1[a] * w;
        const double dn = fx::exp(-y);
        C.nu[a] = nu;
        C.y[a]  = y;
        C.q[a]  = q;
        C.qe[a] = C.A2[a] * w;
        C.dn[a] = dn;
#pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            const double g = P->g[a][s];
            above          = above || g > 1.;
            C.g[a][s]      = g;
            C.vA[a][s]     = q * g;
            C.vE[a][s]     = q * dn * (nbb ? 1. : 1. - g);
        }
    }
    return above;
}

// Adds the rows' contributions of this thread to the 16 moments.  The kernel of
// species 0 (2) at (a, b) is e0 K(a, b) + e1 K(b, a) (x0, x1); species 1 and 3
// exchange K(a, b) and K(b, a) (kernel_pair.hpp:200-216).  SYM: one symmetric
// kernel for all species.  ABS: sums of |term| of the emission moments alone.
template <bool SYM, bool ABS, int NT>
__device__ __forceinline__ void cell_row_sums(const CellNodes<NT>& C, int M, bool stim, double e0,
                                              double e1, double x0, double x1, double* acc)
{
    const int h = C.splits;
    for (int t = threadIdx.x; t < M * h; t += NT)
    {
        const int part = t / M, a = t - part * M;
        const int b0 = part * M / h, b1 = (part + 1) * M / h;
        double F[2][4], G[2][4];
#pragma unroll
        for (int s = 0; s < 4; ++s)
            F[0][s] = F[1][s] = G[0][s] = G[1][s] = 0.;
        for (int b = b0; b < b1; ++b)
        {
            const double k = C.K[a][b];
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                const double v = ABS ? fabs(C.vE[b][s]) : C.vE[b][s];
                F[0][s]        = fma(k, v, F[0][s]);
                if (!ABS)
                    G[0][s] = fma(k, C.vA[b][s], G[0][s]);
            }
            if (!SYM)
            {
                const double kt = C.K[b][a];
#pragma unroll
                for (int s = 0; s < 4; ++s)
                {
                    const double v = ABS ? fabs(C.vE[b][s]) : C.vE[b][s];
                    F[1][s]        = fma(kt, v, F[1][s]);
                    if (!ABS)
                        G[1][s] = fma(kt, C.vA[b][s], G[1][s]);
                }
            }
        }
        const double q = C.q[a], qe = C.qe[a], dn = C.dn[a];
#pragma unroll
        for (int s = 0; s < 4; ++s)
        {
            const int ps    = s ^ 1, o = s & 1;
            const double c0 = s < 2 ? e0 : x0, c1 = s < 2 ? e1 : x1;
            const double Fs = dn * (SYM ? F[0][ps] : fma(c0, F[o][ps], c1 * F[1 - o][ps]));
            const double g  = C.g[a][s];
            if (ABS)
            {
                const double m = stim ? Fs : fabs(1. - g) * Fs;
                acc[s]     = fma(q, m, acc[s]);
                acc[8 + s] = fma(qe, m, acc[8 + s]);
                continue;
            }
            const double Gs = SYM ? G[0][ps] : fma(c0, G[o][ps], c1 * G[1 - o][ps]);
            const double em = stim ? Fs : (1. - g) * Fs;
            const double ab = g * (stim ? Fs + Gs : Gs);
            acc[s]      = fma(q, em, acc[s]);
            acc[4 + s]  = fma(q, ab, acc[4 + s]);
            acc[8 + s]  = fma(qe, em, acc[8 + s]);
            acc[12 + s] = fma(qe, ab, acc[12 + s]);
        }
    }
}

// Totals over the first NT of a CTA's NTW threads: lane l of a warp holds that of moment sum_index(l).
template <int NTW, int NT>
__device__ __forceinline__ double cell_total(CellNodes<NT>& C, double* acc, int slot)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double v = warp_sum16(acc, lane);
    if ((NTW == NT || wid < NT / 32) && !(lane & 1))
        C.red[slot][wid][sum_index(lane)] = v;
    __syncthreads();
    double t = C.red[slot][0][sum_index(lane)];
#pragma unroll
    for (int w = 1; w < NT / 32; ++w)
        t += C.red[slot][w][sum_index(lane)];
    return t;
}

// Node tables of the mixed pair phase: y = nu/T as double-float and
// e^{y - |eta|/2} (e^{Lref} = its product over the two nodes when |eta| >= s).
struct PairTab32
{
    float yh[kMaxM], yl[kMaxM];
    double eh[kMaxM];
};

// Fermi integrals of the FP64 pair kernel at the nodes, scaled as Psi needs
// them: 120 F_1, 120 F_2, 40 F_3, 20 F_4, 4 F_5 at eta -+ y; 1 / y^2.
struct PairTab64
{
    double m[kMaxM][5], p[kMaxM][5], iy2[kMaxM];
};

template <bool MIXED>
struct PairSmem
{
    CellNodes<kCellThreads> C;
    alignas(16) unsigned char tab[MIXED ? sizeof(PairTab32) : sizeof(PairTab64)];
};

// e+e- pair phase.  MIXED: cells from the FP32 integral (bnsn_pair32.cuh); the
// sums and the magnitudes of their terms are written to the record (PairMixed).
// The pair kernels are non-negative and so are the absorption terms (em + am =
// em (1 + g (e^s - 1)) >= 0), so only the emission terms, through 1 - g < 0, can
// carry the opposite sign.  !MIXED: the FP64 kernel (kernel_pair.hpp); with
// redo_only the mixed path's second pass over the points the final kernel
// marked (predo), whose pair part of s2d it replaces; that pass computes its
// Fermi-integral tables itself.
// 8,192 points, n = 20: FP64 2.95 -> 1.35 ms, mixed with its redo pass 2.46 ->
// 1.52 ms; one point, n = 10: 74 -> 23 us.
template <bool MIXED, int NTW>
__device__ __forceinline__ void pair_points(PairSmem<MIXED>& S, const OpacityLaunch& L,
                                            int64_t p0, int64_t np, double* __restrict__ scratch,
                                            int redo_only)
{
    CellNodes<kCellThreads>& C = S.C;
    PairTab32& X = *reinterpret_cast<PairTab32*>(S.tab); // MIXED
    PairTab64& W = *reinterpret_cast<PairTab64*>(S.tab); // !MIXED
    const int M     = 2 * L.n2;
    const int ncell = L.ncell;
    const bool nbb = L.neglect_blocking != 0, stim = L.stim != 0;
    bool ready = false; // launch constants staged

    for (int64_t q = blockIdx.x; q < np; q += gridDim.x)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        if (!MIXED && redo_only && pair_mixed(P)->predo != 1.)
            continue; // uniform: a point per CTA
        if (!ready)
        {
            cell_constants<false>(C, L);
            ready = true;
        }
        const double T   = L.eos[1][p];
        const double eta = L.eos[7][p] / T;
        __syncthreads(); // the previous point's readers are done
        const bool above = __syncthreads_or(cell_nodes(C, P, M, nbb, !MIXED));
        const int a0 = threadIdx.x;
        if (a0 < M)
        {
            const double y = C.y[a0];
            if (MIXED)
            {
                const dfm::df yd = dfm::from_double(y);
                X.yh[a0] = yd.hi;
                X.yl[a0] = yd.lo;
                X.eh[a0] = fx::exp(y - 0.5 * fabs(eta));
            }
            else
                W.iy2[a0] = 1. / (y * y);
        }
        if (!MIXED)
        {
            for (int qq = threadIdx.x; qq < 2 * M; qq += NTW)
            {
                const int a = qq >> 1;
                double f[5];
                if (redo_only) // the tables the mixed prelude left out
                    fdi_orders<1, 5>(qq & 1 ? eta + C.y[a] : eta - C.y[a], f);
                else
                {
#pragma unroll
                    for (int k = 0; k < 5; ++k)
                        f[k] = qq & 1 ? P->fp[a][k] : P->fm[a][k];
                }
                pair_scale(f, qq & 1 ? W.p[a] : W.m[a]);
            }
        }
        __syncthreads();
        const dfm::df ETA = dfm::from_double(eta);
        const double T2   = T * T;
        const double f40 = 40. * P->fe[0][3], f20 = 20. * P->fe[0][4];
        // em = Phi T^2 / 2 (alpha1^2 Psi(y, z) + alpha2^2 Psi(z, y)) / (1 - e^s), ab = e^s em
        const double sc = MIXED ? 0.5 * k::PairPhi * T2 * (T2 * T2) / 15.
                                : -0.5 * k::PairPhi * T2 / 15.;
        for (int c = threadIdx.x; c < ncell; c += NTW)
        {
            const uint32_t ab = C.cells[c];
            const int a = ab & 0xffu, b = ab >> 8;
            double k0 = 0., k1 = 0.;
            if (MIXED)
                pair32::absorption_q(dfm::df{X.yh[a], X.yl[a]}, dfm::df{X.yh[b], X.yl[b]},
                                     X.eh[a], X.eh[b], ETA, sc, &k0, &k1);
            else
            {
                const double y = C.y[a], z = C.y[b];
                if (!(eta - y - z > 200.))
                {
                    pair_psi_scaled(W.m[a], W.p[a], W.m[b], W.p[b], eta, y, z, f40, f20, &k0,
                                    &k1);
                    const double f =
                        sc * (W.iy2[a] * W.iy2[b]) * fx::rcp(1. - C.dn[a] * C.dn[b]);
                    k0 *= f;
                    k1 *= f;
                }
            }
            C.K[a][b] = k0;
            if (a != b)
                C.K[b][a] = k1;
        }
        __syncthreads();
        constexpr double e0 = k::PairA1e * k::PairA1e, e1 = k::PairA2e * k::PairA2e;
        constexpr double x0 = k::PairA1x * k::PairA1x, x1 = k::PairA2x * k::PairA2x;
        double acc[16];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
            acc[kk] = 0.;
        if (NTW == kCellThreads || threadIdx.x < kCellThreads)
            cell_row_sums<false, false>(C, M, stim, e0, e1, x0, x1, acc);
        const double tot = cell_total<NTW>(C, acc, 0);
        double mag       = fabs(tot);
        if (MIXED && above)
        {
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
                acc[kk] = 0.;
            cell_row_sums<false, true>(C, M, stim, e0, e1, x0, x1, acc);
            const double m = cell_total<NTW>(C, acc, 1);
            if (!(sum_index(threadIdx.x & 31) & 4))
                mag = m;
        }
        if (threadIdx.x < 32 && !(threadIdx.x & 1))
        {
            PairMixed* Y  = pair_mixed(P);
            const int idx = sum_index(threadIdx.x);
            if (MIXED)
            {
                P->s2d[idx]   = tot;
                Y->spair[idx] = tot;
                Y->pmag[idx]  = mag;
            }
            else if (redo_only)
                P->s2d[idx] = P->s2d[idx] - Y->spair[idx] + tot;
            else
                P->s2d[idx] = tot;
            if (MIXED && threadIdx.x == 0)
                Y->predo = 0.;
        }
    }
}

template <bool MIXED, bool MULTI = false, int NTW = kCellThreads>
__global__ void __launch_bounds__(NTW)
    grey_pair_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                     int64_t np, double* __restrict__ scratch, int redo_only)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    if (MULTI && !L.use_pair)
        return; // a group without pair (uniform over the CTA)
    __shared__ PairSmem<MIXED> S;
    pair_points<MIXED, NTW>(S, L, p0, np, scratch, redo_only);
}

// ---------------------------------------------------------------------------
// Bremsstrahlung in FP64 (kernel_brem_HR98.hpp, _BRT06.hpp, _GP19.hpp): the cells'
// absorption kernels (emission is K e^{-(w + w')/T}) and the row sums of the cell
// phases.  IMPL: 0 HR98, 1 BRT06, 2 GP19.
// ---------------------------------------------------------------------------

template <int IMPL>
struct Brem64Extra
{
};
template <>
struct Brem64Extra<0>
{
    Hr98Cell hc;
    Hr98Point hr;
};
template <>
struct Brem64Extra<2>
{
    Gp19Record r;
    double p[2][kGp19MaxW];
    Gp19Axis axis;
};

template <int IMPL, int NT>
struct Brem64Smem
{
    CellNodes<NT> C;
    Brem64Extra<IMPL> X;
};

// Launch constants (once per CTA; brem64_point's first barrier orders them).
template <int IMPL, int NT>
__device__ __forceinline__ void brem64_constants(Brem64Smem<IMPL, NT>& S, const OpacityLaunch& L)
{
    cell_constants<true>(S.C, L);
    if constexpr (IMPL == 2)
    {
        if (L.gp19.d3 <= kGp19MaxW)
            for (int k = threadIdx.x; k < L.gp19.d3; k += NT)
                gp19_axis_entry(S.X.axis, L.gp19.logw, L.gp19.d3, k);
    }
}

// The brem sums of a point, by the CTA's threads (the row sums by the first NT): lane l of each warp returns the
// total of moment sum_index(l).
template <int NTW, int IMPL, int NT>
__device__ __forceinline__ double brem64_point(Brem64Smem<IMPL, NT>& S, const OpacityLaunch& L,
                                               PointTab* P, int64_t p)
{
    CellNodes<NT>& C = S.C;
    const int M      = 2 * L.n2;
    const double T   = L.eos[1][p];
    __syncthreads(); // the previous point's readers are done
    cell_nodes(C, P, M, L.neglect_blocking != 0, true);
    bool fast = true; // HR98: every cell within hr98_absorption's range
    if constexpr (IMPL == 0)
    {
        for (int k = threadIdx.x; k < (int)(sizeof(Hr98Point) / sizeof(double)); k += NTW)
            ((double*)&S.X.hr)[k] = ((const double*)&P->hr)[k];
        __syncthreads();
        if (threadIdx.x < 4)
            hr98_cell_from(S.X.hr, threadIdx.x, &S.X.hc);
        const bool out = threadIdx.x < M &&
                         !(C.y[threadIdx.x] > 1e-6 && C.y[threadIdx.x] < 4e4);
        fast = !__syncthreads_or(out);
        fast = fast && S.X.hc.fast;
    }
    bool prof = false;
    if constexpr (IMPL == 2)
    {
        prof = L.gp19.d3 <= kGp19MaxW;
        if (prof)
        {
            for (int k = threadIdx.x; k < (int)(sizeof(Gp19Record) / sizeof(double)); k += NTW)
                ((double*)&S.X.r)[k] = ((const double*)gp19_record(P))[k];
            __syncthreads();
            const Gp19Table G = gp19_table(L);
            const int np19    = S.X.r.pt.regime >= 2 ? 2 : 1;
            for (int e = threadIdx.x; e < np19 * G.d3; e += NTW)
            {
                const int pr = e / G.d3, l = e - pr * G.d3;
                S.X.p[pr][l] = gp19_profile_eval(G, S.X.r.cor[pr], l);
            }
        }
    }
    __syncthreads();
    for (int c = threadIdx.x; c < L.ncell; c += NTW)
    {
        const uint32_t ab = C.cells[c];
        const int a = ab & 0xffu, b = ab >> 8;
        double K, em;
        if constexpr (IMPL == 0)
        {
            if (fast)
                K = hr98_absorption(S.X.hc, C.y[a] + C.y[b], C.dn[a] * C.dn[b]);
            else
                hr98_kernel(S.X.hr, C.nu[a], C.nu[b], &em, &K);
        }
        else if constexpr (IMPL == 1)
            K = P->brt06_pre * brt06_shape(0.5 * (C.y[a] + C.y[b]));
        else
        {
            const Gp19Table G = gp19_table(L);
            if (prof)
            {
                const double w = fmax(fmin(C.nu[a] + C.nu[b], G.w[G.d3 - 1]), G.w[0]);
                K = gp19_profile_absorption(S.X.r.pt, S.X.p, S.X.axis, G.d3, w);
            }
            else
                gp19_kernel(G, L.eos[0][p], L.eos[2][p], T, C.nu[a], C.nu[b], &em, &K);
        }
        C.K[a][b] = K;
        C.K[b][a] = K;
    }
    __syncthreads();
    double acc[16];
#pragma unroll
    for (int kk = 0; kk < 16; ++kk)
        acc[kk] = 0.;
    if (NTW == NT || threadIdx.x < NT)
        cell_row_sums<true, false>(C, M, L.stim != 0, 1., 0., 1., 0., acc);
    return cell_total<NTW>(C, acc, 0);
}

// Every point (the plain path), or with redo_only the points the mixed path's
// final kernel marked (bredo = 1), whose brem part of s2d it replaces.
// 8,192 points: HR98 n = 10 1.40 -> 0.44 ms, GP19 n = 20 2.66 -> 0.84 ms, BRT06 n = 10
// 0.65 -> 0.26 ms.
template <int NTW, int IMPL>
__device__ __forceinline__ void brem_points(Brem64Smem<IMPL, kCellThreads>& S,
                                            const OpacityLaunch& L, int64_t p0, int64_t np,
                                            double* __restrict__ scratch, int add, int redo_only)
{
    bool ready = false;
    for (int64_t q = blockIdx.x; q < np; q += gridDim.x)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        if (redo_only && P->bredo != 1.)
            continue; // uniform: a point per CTA
        if (!ready)
        {
            brem64_constants(S, L);
            ready = true;
        }
        const double tot = brem64_point<NTW>(S, L, P, p);
        if (threadIdx.x < 32 && !(threadIdx.x & 1))
        {
            const int idx     = sum_index(threadIdx.x);
            const double base = add ? (redo_only ? P->s2d[idx] - P->sbrem[idx] : P->s2d[idx]) : 0.;
            P->s2d[idx]   = base + tot;
            P->sbrem[idx] = tot;
            P->bmag[idx]  = 0.;
        }
    }
}

template <int IMPL, bool MULTI = false, int NTW = kCellThreads>
__global__ void __launch_bounds__(NTW)
    grey_brem_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                     int64_t np, double* __restrict__ scratch, int add, int redo_only)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
        if (!L.use_brem || L.brem_impl != IMPL)
            return; // another brem variant's launch serves this group
        add = L.use_pair;
    }
    __shared__ Brem64Smem<IMPL, kCellThreads> S;
    brem_points<NTW>(S, L, p0, np, scratch, add, redo_only);
}

// Per-warp GP19 state of the FP32 brem kernel.
struct Gp19Warp
{
    Gp19Record r;
    double p[2][kGp19MaxW];
    float pf[2][kGp19MaxW];
};

// Shared memory of the FP32 brem kernel (later the FP64 one's).
template <int IMPL>
struct Brem32Smem
{
    static constexpr int kWF = IMPL == 2 ? kGp19MaxW : 1;
    dfm::df A1d[kMaxM], A2d[kMaxM];
    uint32_t cells[kMaxCells];
    CellTab ct[kWarps];
    CellTab32 c32[kWarps];
    Gp19Warp gw[IMPL == 2 ? kWarps : 1];
    double lw[kWF], wax[kWF], iw[kWF];
    float lwf[kWF], idl[kWF];
};

// Bremsstrahlung of the mixed path: FP32 cells (bnsn_fp32.cuh), a point per warp.
// Points with the GP19 high-T extrapolation (which differences two table values),
// with tables too long for profiles, or whose cells the other reactions cancel
// are marked (bredo = 2) and evaluated in FP64 by the whole CTA at the end.
template <int IMPL, bool MULTI = false>
__global__ void __launch_bounds__(kWarps * 32, 3)
    grey_brem32_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                     int64_t np, double* __restrict__ scratch, int add)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    if (MULTI)
    {
        if (!L.use_brem || L.brem_impl != IMPL)
            return; // another brem variant's launch serves this group
        add = L.use_pair;
    }
    constexpr size_t kBytes = sizeof(Brem32Smem<IMPL>) > sizeof(Brem64Smem<IMPL, kWarps * 32>)
                                  ? sizeof(Brem32Smem<IMPL>)
                                  : sizeof(Brem64Smem<IMPL, kWarps * 32>);
    __shared__ __align__(16) unsigned char s_raw[kBytes];
    Brem32Smem<IMPL>& S = *reinterpret_cast<Brem32Smem<IMPL>*>(s_raw);
    const Gp19Table G19 = gp19_table(L);
    const bool prof = IMPL == 2 && G19.d3 <= kGp19MaxW;
    for (int k = threadIdx.x; k < kMaxM; k += blockDim.x)
    {
        S.A1d[k] = dfm::from_double(L.A1[k]);
        S.A2d[k] = dfm::from_double(L.A2[k]);
    }
    for (int k = threadIdx.x; k < L.ncell; k += blockDim.x)
        S.cells[k] = L.cells[k];
    if (IMPL == 2 && prof)
        for (int k = threadIdx.x; k < G19.d3; k += blockDim.x)
        {
            S.lw[k]  = G19.logw[k];
            S.lwf[k] = (float)G19.logw[k];
            S.wax[k] = G19.w[k];
            S.iw[k]  = 1. / G19.w[k];
            S.idl[k] = k + 1 < G19.d3 ? (float)(1. / (G19.logw[k + 1] - G19.logw[k])) : 0.f;
        }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wid  = threadIdx.x >> 5;
    CellTab& C     = S.ct[wid];
    const int M    = 2 * L.n2;
    const bool nbb = L.neglect_blocking != 0;
    const int64_t qstep = (int64_t)gridDim.x * kWarps;
    const double wmin = IMPL == 2 ? G19.w[0] : 0., wmax = IMPL == 2 ? G19.w[G19.d3 - 1] : 0.;

    for (int64_t q = (int64_t)blockIdx.x * kWarps + wid; q < np; q += qstep)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        const double T  = L.eos[1][p];
        Gp19Warp& GW    = S.gw[IMPL == 2 ? wid : 0];
        __syncwarp();
        if (IMPL == 2)
        {
            if (prof)
                warp_copy((double*)&GW.r, (const double*)gp19_record(P),
                          sizeof(Gp19Record) / sizeof(double), lane);
            __syncwarp();
            if (!prof || GW.r.pt.regime == 3 || GW.r.pt.regime == 5)
            {
                if (lane == 0)
                    P->bredo = 2.;
                continue; // uniform: one point per warp
            }
        }
        load_cell_tab(C, P, M, lane);
        if (IMPL == 0 && lane < 4)
            fp32::hr98_mixed_part(P->hr, lane, &C.hm);
        if (IMPL == 2)
        {
            const int np19 = (GW.r.pt.regime >= 2) ? 2 : 1;
            for (int e = lane; e < np19 * G19.d3; e += 32)
            {
                const int pr = e / G19.d3, l = e - pr * G19.d3;
                const double v = gp19_profile_eval(G19, GW.r.cor[pr], l);
                GW.p[pr][l]  = v;
                GW.pf[pr][l] = (float)v;
            }
        }
        __syncwarp();
        double acc[16];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
            acc[kk] = 0.;
        {
            CellTab32& D = S.c32[wid];
            fill_tab32(D, C, M, lane);
            __syncwarp();
            double scale = (T * T) * (T * T);
            float thr = 0.f, lt2 = 0.f;
            if (IMPL == 0)
                scale *= C.hm.outer;
            else if (IMPL == 1)
                scale *= C.brt06_pre;
            else
            {
                scale *= 3. * GW.r.pt.C;
                thr = (float)(1e-30 / GW.r.pt.C);
                lt2 = (float)fx::log2(T * 0.5);
            }
            Acc32 A;
            A.clear();
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
                A.mag[kk] = 0.f;
            int pending = 0;
            for (int c = lane; c < L.ncell; c += 32)
            {
                const uint32_t ab = S.cells[c];
                const int a = ab & 0xffffu, b = ab >> 16;
                // x = (nu_a + nu_b) / T as hi + lo (accurate exponent)
                const dfm::df xs = dfm::add(dfm::df{D.yh[a], D.yl[a]}, dfm::df{D.yh[b], D.yl[b]});
                const float ex = expf(-xs.hi) * (1.f - xs.lo);
                float Kab;
                bool slow = false;
                if (IMPL == 0)
                    Kab = fp32::hr98_shape(C.hm, xs.hi, xs.lo);
                else if (IMPL == 1)
                {
                    // BRT06 (kernel_brem_BRT06.hpp:24-69): ab = pre K_1(x) e^{x} / x,
                    // x = (nu_a + nu_b) / 2T; em = ab e^{-2x}
                    const float xh = 0.5f * (xs.hi + xs.lo);
                    Kab            = fp32::bessk1e(xh) / xh;
                }
                else
                {
                    double wv = C.nu[a] + C.nu[b];
                    wv        = wv > wmax ? wmax : (wv < wmin ? wmin : wv);
                    float tw;
                    const int l = gp19_bracket32(wv, S.lwf, S.wax, S.iw, S.idl, G19.d3, &tw);
                    const float v0 = GW.pf[0][l] + tw * (GW.pf[0][l + 1] - GW.pf[0][l]);
                    if (GW.r.pt.regime <= 1)
                        Kab = v0;
                    else
                    {
                        const float v1 = GW.pf[1][l] + tw * (GW.pf[1][l + 1] - GW.pf[1][l]);
                        Kab = v0 * exp2f(log2f(v1 / v0) * lt2);
                        // regime 2 clips k2, k4 and s at 1e-30 (rare: exact FP64 cell)
                        slow = GW.r.pt.regime == 2 && (v0 < thr || v1 < thr || Kab < thr);
                    }
                    Kab = fabsf(Kab);
                }
                float Kem = Kab * ex;
                if (IMPL == 2 && slow)
                {
                    const double nua = C.nu[a], nub = C.nu[b];
                    double w = nua + nub;
                    w        = w > wmax ? wmax : (w < wmin ? wmin : w);
                    double tw;
                    const int l = bracket_sorted<double>(log(w), S.lw, G19.d3, &tw);
                    const double v0 = GW.p[0][l] * (1. - tw) + GW.p[0][l + 1] * tw;
                    const double v1 = GW.p[1][l] * (1. - tw) + GW.p[1][l + 1] * tw;
                    double em, abv;
                    gp19_cell(GW.r.pt, v0, v1, w, nua + nub, &em, &abv);
                    Kab = (float)(abv / (3. * GW.r.pt.C));
                    Kem = (float)(em / (3. * GW.r.pt.C));
                }
                const dfm::df yab = dfm::mul(dfm::df{D.yh[a], D.yl[a]}, dfm::df{D.yh[b], D.yl[b]});
                const dfm::df w4  = dfm::mul(yab, yab); // (y_a y_b)^2
                const float P1    = cell_weight(w4, S.A1d[a], S.A1d[b]);
                const float P2    = cell_weight(w4, S.A2d[a], S.A1d[b]);
                if (L.stim)
                    add_cell32<true>(A, Kem, Kab, D.g[a], D.gm[a], D.g[b], D.gm[b], nbb, P1, P2);
                else
                    add_cell32<false>(A, Kem, Kab, D.g[a], D.gm[a], D.g[b], D.gm[b], nbb, P1, P2);
                if (a != b)
                {
                    const float P2r = cell_weight(w4, S.A2d[b], S.A1d[a]);
                    if (L.stim)
                        add_cell32<true>(A, Kem, Kab, D.g[b], D.gm[b], D.g[a], D.gm[a], nbb, P1,
                                         P2r);
                    else
                        add_cell32<false>(A, Kem, Kab, D.g[b], D.gm[b], D.g[a], D.gm[a], nbb, P1,
                                          P2r);
                }
                if (++pending == 4)
                {
#pragma unroll
                    for (int kk = 0; kk < 16; ++kk)
                        acc[kk] += (double)A.v[kk];
                    A.clear();
                    pending = 0;
                }
            }
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
                acc[kk] = acc[kk] + (double)A.v[kk];
            // cells of both signs (occupation above 1 makes 1 - g negative), or
            // a brem sum cancelling the pair sum or the beta rates: this point
            // goes to FP64.  Each lane checks the moment whose total it holds.
            double mg[16];
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
                mg[kk] = (double)A.mag[kk];
            const int idx      = sum_index(lane);
            const double tot   = warp_sum16(acc, lane) * scale;
            const double mag   = warp_sum16(mg, lane) * scale;
            const double base  = add ? P->s2d[idx] : 0.;
            const double other =
                beta_in_sum_unit(P, T, L.eos[7][p] / T, L.use_abs_em, false, idx) + base;
            const bool redo = __any_sync(0xffffffffu,
                                         mag > 0. && mag > kMaxCancelBrem * fabs(tot + other));
            if (lane == 0)
                P->bredo = redo ? 2. : 0.;
            if (!redo && !(lane & 1))
            {
                P->s2d[idx]   = base + tot;
                P->sbrem[idx] = tot;
                P->bmag[idx]  = mag;
            }
        }
    }
    // the marked points of this CTA
    Brem64Smem<IMPL, kWarps * 32>& S64 = *reinterpret_cast<Brem64Smem<IMPL, kWarps * 32>*>(s_raw);
    __syncthreads(); // the FP32 tables' readers are done
    bool ready = false;
    for (int64_t qb = (int64_t)blockIdx.x * kWarps; qb < np; qb += qstep)
        for (int64_t q = qb; q < qb + kWarps && q < np; ++q)
        {
            PointTab* P = (PointTab*)(scratch + q * kTabWords);
            if (P->bredo != 2.)
                continue; // uniform
            if (!ready)
            {
                brem64_constants(S64, L);
                ready = true;
            }
            const double tot = brem64_point<kWarps * 32>(S64, L, P, L.pidx ? L.pidx[p0 + q] : p0 + q);
            if (threadIdx.x < 32 && !(threadIdx.x & 1))
            {
                const int idx = sum_index(threadIdx.x);
                P->s2d[idx]   = (add ? P->s2d[idx] : 0.) + tot;
                P->sbrem[idx] = tot;
                P->bmag[idx]  = 0.;
            }
        }
}

// ---------------------------------------------------------------------------
// NES / NPS (m1_opacities.hpp:864-1057, integration.hpp:687-768)
// ---------------------------------------------------------------------------
struct NepsTab
{
    double fe[2][6];
    double fd0[2];
};

// The mixed path's NES runs three launches per chunk:
//   grey_nes_fast_kernel  FP32 kernel integrals (bnsn_nes32.cuh); flags a
//                 point 1 when its sums cancel (terms of both signs, or
//                 negative pair + brem sums) and 2 when it leaves the FP32
//                 range envelope;
//   grey_nes_list_kernel  the flagged points' list;
//   grey_nes64_kernel     FP64 items of the listed points, a point per CTA (the plain
//                 path runs it over every point).
// A pass with every product in double-float over the points flagged 1, with FP64 for
// the sums that cancel beyond 1e5, took 128 us of 1,001 points at n = 6 (one CTA per point
// running long chains), now 38, and 0.42 ms of 8,192 at n = 20, now 0.13.

// The list in the mixed path's record words of F_k(eta + nu/T), which it leaves free:
// word 0 of record 0 its length, then its entries, 400 a record.
__device__ __forceinline__ int* nes_list(double* scratch, int64_t k)
{
    constexpr int per = 2 * 5 * kMaxM;
    return (int*)&((PointTab*)(scratch + k / per * kTabWords))->fp[0][0] + k % per;
}

template <bool MULTI = false>
__global__ void __launch_bounds__(256)
    grey_nes_list_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t np,
                         double* __restrict__ scratch)
{
    if (MULTI)
    {
        if (!GA.Ls[blockIdx.z].use_inel)
            return;
        np      = GA.gc[blockIdx.z].np;
        scratch = GA.gc[blockIdx.z].ws;
    }
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool in   = q < np && ((PointTab*)(scratch + q * kTabWords))->neps_fp64 != 0.;
    const uint32_t m = __ballot_sync(0xffffffffu, in);
    if (m == 0u)
        return;
    const int lane = threadIdx.x & 31;
    int first      = 0;
    if (lane == 0)
        first = atomicAdd(nes_list(scratch, 0), __popc(m));
    first = __shfl_sync(0xffffffffu, first, 0);
    if (in)
        *nes_list(scratch, 1 + first + __popc(m & ((1u << lane) - 1u))) = (int)q;
}


// ---------------------------------------------------------------------------
// NES/NPS in FP64 (kernel_nes.hpp:50-359; the item sums of
// m1_opacities.hpp:864-1057 and integration.hpp:687-768).
//
// MezzacappaIntOut is antisymmetric, linear in its couplings (nes_bracket), and an
// item's energies in units of T do not depend on the point; the weight (nu
// nubar)^2 of the item cancels the bracket's 1 / P^2.  So a lepton takes three sets
// of Fermi integrals and 17 FP64 operations, where the four species and two
// directions separately took 16 evaluations of the bracket with a division each
// (~560 instructions); both leptons' A and B combine into the four species'
// kernels afterwards, R(w', w) = -R(w, w') costs nothing, and the NEPSExpFunc
// factors, weights and w^0.6 sit in the CTA's item table.
// The items follow the host's order of ascending w', which keeps a warp's lanes in
// the same regime of the Fermi integrals.
//
// Bound by the FP64 pipe (~200 operations an item) beside the integer work of
// its exponentials and Fermi integrals.  Two warps share a point in 16-warp CTAs
// (the 38 KB item table serves 8 points; one warp per point left the last of
// 3.4 waves over 8,192 points 60% empty), or (WIDE) eight in 8-warp CTAs: the
// mixed path's few flagged points, and launches with fewer points than the chip
// has warps to fill.  8,192 points, n = 20: 5.41 -> 3.69 ms.
// ---------------------------------------------------------------------------

template <bool WIDE>
struct Nes64Smem
{
    static constexpr int kItems = kMaxQ * kMaxQ * 2;
    static constexpr int kNW    = WIDE ? 8 : 16;  // warps of the CTA
    static constexpr int kWPP   = WIDE ? 8 : 2;   // warps per point
    static constexpr int kPts   = kNW / kWPP;
    double w[kItems], wp[kItems];   // w, w'
    double ka[kItems], m[kItems];   // 24 weight e / (1 - e), 24 weight
    double wc[kItems], wpc[kItems]; // w^0.6, w'^0.6
    Occ64 occ[kPts][4];
    double fe[kPts][2][6], fd0[kPts][2];
    double red[kPts][2][16];
    int twin[kPts];
    double terms[WIDE ? 16 : 1][WIDE ? kNW * 32 : 1]; // EM1, AB1, EM2, AB2 of a round's items
};

template <bool WIDE>
__device__ __forceinline__ void nes64_points(Nes64Smem<WIDE>& S, const OpacityLaunch& L,
                                             int64_t p0, int64_t np,
                                             double* __restrict__ scratch, int flagged)
{
    using Smem = Nes64Smem<WIDE>;
    constexpr int kStride = Smem::kWPP * 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int slot = wid / Smem::kWPP, wsub = wid - slot * Smem::kWPP;
    const int n2 = L.n2, nn2 = n2 * n2, nit = 2 * nn2;
    const bool nbb = L.neglect_blocking != 0, stim = L.stim != 0;
    // the warps of a point (every thread of them runs the same iterations)
    const auto point_sync = [&]() {
        if (WIDE)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(kStride) : "memory");
    };
    const auto make_table = [&]() {
        // w = c x_i (1 -+ x_j) for r = 0 and c (1 -+ x_j) / x_i for r = 1
        // (m1_opacities.hpp:880-905), c = 2 x 2.182
        constexpr double c = 2. * k::TempMultiple;
        for (int k = threadIdx.x; k < nit; k += blockDim.x)
        {
            const int it  = L.nes_order[k];
            const int r   = it >= nn2;
            const int rem = it - r * nn2;
            const int i = rem / n2, j = rem - (rem / n2) * n2;
            const double xi = L.x2[i], xj = L.x2[j];
            const double w  = r ? c * (1. - xj) / xi : c * xi * (1. - xj);
            const double wp = r ? c * (1. + xj) / xi : c * xi * (1. + xj);
            const double e1 = -expm1(-(wp - w)); // 1 - e
            const double m  = 24. * ((r ? L.wx3[i] : L.wx[i]) * L.w2[j]);
            S.w[k]   = w;
            S.wp[k]  = wp;
            S.m[k]   = m;
            S.ka[k]  = m * (fx::exp(w - wp) / e1);
            S.wc[k]  = fx::pow(w, k::CF);
            S.wpc[k] = fx::pow(wp, k::CF);
        }
    };
    bool table = !WIDE;
    if (!WIDE)
    {
        make_table();
        __syncthreads();
    }
    const bool listed = WIDE && flagged; // the list's points, else all
    const int64_t nw  = listed ? *nes_list(scratch, 0) : np;
    for (int64_t k = (int64_t)blockIdx.x * Smem::kPts + slot; k < nw;
         k += (int64_t)gridDim.x * Smem::kPts)
    {
        const int64_t q = listed ? *nes_list(scratch, 1 + k) : k;
        const int64_t p = L.pidx ? L.pidx[p0 + q] : p0 + q;
        PointTab* P     = (PointTab*)(scratch + q * kTabWords);
        if (!table)
        {
            make_table(); // before the point's first barrier below
            table = true;
        }
        const double T = L.eos[1][p], mu_e = L.eos[7][p];
        point_sync(); // the previous point's readers are done
        if (wsub == 0)
        {
            const Distr& d = P->d;
            if (lane < 4)
                occ64_from(d, lane, T, &S.occ[slot][lane]);
            else if (lane >= 16 && lane < 28)
                (&S.fe[slot][0][0])[lane - 16] = (&P->fe[0][0])[lane - 16];
            else if (lane >= 28 && lane < 30)
                S.fd0[slot][lane - 28] = P->fd0[lane - 28];
            else if (lane == 30) // heavy-lepton neutrinos evolved as one species
                S.twin[slot] = species_twins(d);
        }
        point_sync();
        const Occ64* occ  = S.occ[slot];
        const bool common = occ[0].cf == k::CF && occ[1].cf == k::CF && occ[2].cf == k::CF &&
                            occ[3].cf == k::CF;
        const int nocc   = S.twin[slot] ? 3 : 4;
        const double pre = k::NepsConst * (T * T), eta_e = mu_e / T;
        double acc[16];
#pragma unroll
        for (int kk = 0; kk < 16; ++kk)
            acc[kk] = 0.;
        // EM1[4], AB1[4], EM2[4], AB2[4] of item it; products are rounded here so
        // that both forms of the kernel add the same numbers
        const auto item_terms = [&](int it, double* o) {
            const double w = S.w[it], wp = S.wp[it];
            const double dl = wp - w;
            double U = 0., V = 0.; // A of e- + B of e+, B of e- + A of e+
#pragma unroll 1
            for (int e = 0; e < 2; ++e)
            {
                const double eta = e ? -eta_e : eta_e, thr = eta * 1e-3;
                const double* fe = S.fe[slot][e];
                double A, B;
                if (w > thr)
                {
                    double a[5], b[5];
                    fx::fd_orders<1, 5, true>(eta - wp, a);
                    fx::fd_orders<1, 5, true>(eta - w, b);
                    nes_bracket(eta, wp, w, dl, a, b, fe, &A, &B);
                }
                else
                    nes_bracket_taylor(eta, wp, w, dl, fe, S.fd0[slot][e], &A, &B);
                U += e ? B : A;
                V += e ? A : B;
            }
            constexpr double bp = k::NepsBPlus, bm = k::NepsBMinus, bz = k::NepsBZero;
            const double zU = bz * U, zV = bz * V;
            const double c[4] = {fma(bp, U, zV), fma(bp, V, zU), fma(bm, U, zV), fma(bm, V, zU)};
            double g[4], gb[4];
            const double wc = S.wc[it], wpc = S.wpc[it];
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                if (s < nocc)
                {
                    g[s]  = occ64_one(occ[s], w, common ? wc : fx::pow(w, occ[s].cf));
                    gb[s] = occ64_one(occ[s], wp, common ? wpc : fx::pow(wp, occ[s].cf));
                }
                else
                {
                    g[s]  = g[2];
                    gb[s] = gb[2];
                }
            }
            const double m = S.m[it], ka = S.ka[it], kb = ka + m;
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                // emission and absorption kernels nu -> nubar; nubar -> nu swaps them
                const double ke = kb * c[s], kk = ka * c[s];
                const double e1 = __dmul_rn(ke, gb[s]), e2 = __dmul_rn(kk, g[s]);
                if (stim)
                {
                    // e + a = e + k (1 - g), the difference of the kernels in one product
                    const double mc = m * c[s];
                    o[s]      = e1;
                    o[8 + s]  = e2;
                    o[4 + s]  = __dmul_rn(g[s], nbb ? e1 + kk : fma(gb[s], mc, kk));
                    o[12 + s] = __dmul_rn(gb[s], nbb ? e2 + ke : fma(-g[s], mc, ke));
                }
                else
                {
                    o[s]      = __dmul_rn(1. - g[s], e1);
                    o[8 + s]  = __dmul_rn(1. - gb[s], e2);
                    o[4 + s]  = __dmul_rn(g[s], nbb ? kk : kk * (1. - gb[s]));
                    o[12 + s] = __dmul_rn(gb[s], nbb ? ke : ke * (1. - g[s]));
                }
            }
        };
        const auto add_terms = [&](int it, const double* o) {
            const double w = S.w[it], wp = S.wp[it];
#pragma unroll
            for (int s = 0; s < 8; ++s) // emission, absorption
            {
                acc[s]     = __dadd_rn(acc[s], __dadd_rn(o[s], o[8 + s]));
                acc[8 + s] = fma(w, o[s], fma(wp, o[8 + s], acc[8 + s]));
            }
        };
        if (!WIDE)
        {
#pragma unroll 1
            for (int it = wsub * 32 + lane; it < nit; it += 64)
            {
                double o[16];
                item_terms(it, o);
                add_terms(it, o);
            }
        }
        else
        {
            // rounds of 256 items; the first two warps add them as the two-warp
            // form does (64 partial sums), so that a point's sums do not depend on
            // the form
#pragma unroll 1
            for (int base = 0; base < nit; base += kStride)
            {
                const int it = base + (int)threadIdx.x;
                if (it < nit)
                {
                    double o[16];
                    item_terms(it, o);
#pragma unroll
                    for (int kk = 0; kk < 16; ++kk)
                        S.terms[kk][threadIdx.x] = o[kk];
                }
                __syncthreads();
                if (wid < 2)
                {
#pragma unroll 1
                    for (int v = threadIdx.x; v < kStride && base + v < nit; v += 64)
                    {
                        double o[16];
#pragma unroll
                        for (int kk = 0; kk < 16; ++kk)
                            o[kk] = S.terms[kk][v];
                        add_terms(base + v, o);
                    }
                }
                __syncthreads();
            }
        }
        if (wsub < 2)
        {
            const double v = warp_sum16(acc, lane);
            if (!(lane & 1))
                S.red[slot][wsub][sum_index(lane)] = v;
        }
        point_sync();
        if (wsub == 0 && !(lane & 1))
        {
            const int idx  = sum_index(lane);
            const double t = S.red[slot][0][idx] + S.red[slot][1][idx];
            P->snes[idx] = t * (pre * ((T * T) * (T * T)) * (idx >= 8 ? T : 1.));
        }
    }
}

template <bool WIDE, bool MULTI = false>
__global__ void __launch_bounds__(Nes64Smem<WIDE>::kNW * 32, WIDE ? 2 : 1)
    grey_nes64_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                      int64_t np, double* __restrict__ scratch, int flagged)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    if (MULTI && !L.use_inel)
        return;
    extern __shared__ __align__(16) unsigned char nes_smem_raw[];
    nes64_points(*reinterpret_cast<Nes64Smem<WIDE>*>(nes_smem_raw), L, p0, np, scratch, flagged);
}

// Pair + brem (blockIdx.y = 0) and NES (1) of small FP64 calls in one launch, a point per
// CTA: they need only the prelude's tables, and each alone leaves most of the chip and of
// its own CTA's latency unused.  One point, n = 10 HR98: the three phases 83 -> 46 us.
template <int IMPL>
__global__ void __launch_bounds__(kCellWide, 2)
    grey_small_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0, int64_t np,
                      double* __restrict__ scratch)
{
    static_assert(Nes64Smem<true>::kNW * 32 == kCellWide, "one CTA size");
    static_assert(sizeof(PairSmem<false>) <= sizeof(Nes64Smem<true>) &&
                      sizeof(Brem64Smem<IMPL, kCellThreads>) <= sizeof(Nes64Smem<true>),
                  "shared memory of the launch");
    extern __shared__ __align__(16) unsigned char nes_smem_raw[];
    if (blockIdx.y == 1)
    {
        nes64_points(*reinterpret_cast<Nes64Smem<true>*>(nes_smem_raw), L, p0, np, scratch, 0);
        return;
    }
    if (L.use_pair)
        pair_points<false, kCellWide>(*reinterpret_cast<PairSmem<false>*>(nes_smem_raw), L, p0, np,
                                      scratch, 0);
    __syncthreads(); // the pair tables' readers are done
    if (L.use_brem)
        brem_points<kCellWide>(*reinterpret_cast<Brem64Smem<IMPL, kCellThreads>*>(nes_smem_raw), L,
                               p0, np, scratch, L.use_pair, 0);
}

// ---------------------------------------------------------------------------
// NES/NPS fast pass of the mixed path (InelasticScattKernels and the grey
// item sums of m1_opacities.hpp:880-905): two warps per point (or a CTA), one item per
// lane, the kernel integrals of bnsn_nes32.cuh in FP32.
// ---------------------------------------------------------------------------

constexpr int kNesWarps = 8;
constexpr int kNesItems = 2 * kMaxQ * kMaxQ;

// One (w, w') item.  w = nu/T and w' = nubar/T depend only on the quadrature
// nodes, so one table per CTA serves every point; the table follows the
// host's item order (ascending max(w, w')), which keeps a warp's lanes on
// items of similar quadrature cost.
struct NesItem
{
    float wh, wl, wph, wpl;     // w, w' as df
    float lwh, lwl, lwph, lwpl; // log w, log w' as df
    float sefa, sefb;           // sign x NEPSExpFunc(w' - w), sign x NEPSExpFunc(w - w')
    float wf;                   // quadrature weight
    float pad;
};

// Data of the point in work.
struct NesPointData
{
    NepsTab N; // F_k(eta) for the FP64 Taylor branches
    nes32::Lepton lep[2];
    NuSpecies sp[4];
    int twin; // species 2 and 3 share one distribution
};

template <bool WIDE>
struct NesSmem
{
    static constexpr int kWPP = WIDE ? kNesWarps : 2; // warps per point
    static constexpr int kPts = kNesWarps / kWPP;
    NesItem items[kNesItems];
    NesPointData pt[kPts];
    static constexpr int kSum = kPts * 64; // partial sums: 64 lanes per point
    uint16_t q[kPts * 2][kNesItems / 2 + 32]; // items (| lepton mask << 14) for the Taylor branches
    float2 dacc[16][kSum]; // per-lane df sums of the 16 moments
    float4 mag[4][kSum];   // per-lane sums of |term|
    double red[kPts][2][2][16];
    float tm[WIDE ? 16 : 1][WIDE ? kNesWarps * 32 : 1]; // terms of a round's items
    uint8_t tmk[WIDE ? kNesWarps * 32 : 1];             // their Taylor mask, bit 2: has terms
};

// One item's terms of the 16 moments: em1..ab2 are R(nu, nubar) and R(nubar, nu)
// with NEPSExpFunc applied, times (w w')^2 (m1_opacities.hpp:880-905).
__device__ __forceinline__ void nes_terms(bool stim, bool nbb, float Wf, float fw, float fwp,
                                          const float* g, const float* gm, const float* gb,
                                          const float* gbm, const float* em1, const float* ab1,
                                          const float* em2, const float* ab2, float* tm)
{
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        const float e1 = em1[s] * gb[s];
        const float a1 = ab1[s] * (nbb ? 1.f : gbm[s]);
        const float e2 = em2[s] * g[s];
        const float a2 = ab2[s] * (nbb ? 1.f : gm[s]);
        float EM1, AB1, EM2, AB2;
        if (stim)
        {
            AB1 = g[s] * (e1 + a1);
            EM1 = e1;
            AB2 = gb[s] * (e2 + a2);
            EM2 = e2;
        }
        else
        {
            AB1 = g[s] * a1;
            EM1 = gm[s] * e1;
            AB2 = gb[s] * a2;
            EM2 = gbm[s] * e2;
        }
        tm[s]      = Wf * (EM1 + EM2);
        tm[4 + s]  = Wf * (AB1 + AB2);
        tm[8 + s]  = Wf * (fw * EM1 + fwp * EM2);
        tm[12 + s] = Wf * (fw * AB1 + fwp * AB2);
    }
}

// Adds them to the sums of (virtual) lane t.
template <class Smem>
__device__ __forceinline__ void nes_accumulate(Smem& S, int t, const float* tm)
{
#pragma unroll
    for (int kk = 0; kk < 16; ++kk)
    {
        const float2 a   = S.dacc[kk][t];
        const dfm::df r  = dfm::add(dfm::df{a.x, a.y}, tm[kk]);
        S.dacc[kk][t]    = make_float2(r.hi, r.lo);
    }
#pragma unroll
    for (int k4 = 0; k4 < 4; ++k4)
    {
        float4 m = S.mag[k4][t];
        m.x += fabsf(tm[4 * k4]);
        m.y += fabsf(tm[4 * k4 + 1]);
        m.z += fabsf(tm[4 * k4 + 2]);
        m.w += fabsf(tm[4 * k4 + 3]);
        S.mag[k4][t] = m;
    }
}

// Two warps share a point, rows of 32 items alternating between them (with a warp
// per point the last of 3.4 waves over 8,192 points ran 60% empty), or (WIDE, for
// launches with fewer points than the chip has warps to fill) all eight.  The 16
// moments' totals and magnitudes are summed so that a lane holds one moment,
// whose cancellation it checks.  8,192 points, n = 20: 2.78 -> 2.45 ms; one point, n =
// 10: 148 -> 58 us.
template <bool WIDE, bool MULTI = false>
__global__ void __launch_bounds__(kNesWarps * 32, 2)
    grey_nes_fast_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA,
                         int64_t p0, int64_t np, double* __restrict__ scratch)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    if (MULTI && !L.use_inel)
        return;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *nes_list(scratch, 0) = 0; // grey_nes_list_kernel fills it
    extern __shared__ __align__(16) unsigned char nes_smem_raw[];
    using Smem   = NesSmem<WIDE>;
    Smem& S      = *reinterpret_cast<Smem*>(nes_smem_raw);
    const int n2 = L.n2, nn2 = n2 * n2, nit = 2 * nn2;
    {
        // w = c x_i (1 -+ x_j) for r = 0 and c (1 -+ x_j) / x_i for r = 1, c = 2 x 2.182
        constexpr double c = 2. * k::TempMultiple;
        const double lc    = log(c);
        for (int k = threadIdx.x; k < nit; k += blockDim.x)
        {
            const int it    = L.nes_order[k];
            const int r     = it >= nn2;
            const int rem   = it - r * nn2;
            const int i     = rem / n2, j = rem - (rem / n2) * n2;
            const double xi = L.x2[i], xj = L.x2[j];
            const double w  = r ? c * (1. - xj) / xi : c * xi * (1. - xj);
            const double wp = r ? c * (1. + xj) / xi : c * xi * (1. + xj);
            const double lw  = lc + (r ? L.l1m[j] - L.lx2[i] : L.lx2[i] + L.l1m[j]);
            const double lwp = lc + (r ? L.l1p[j] - L.lx2[i] : L.lx2[i] + L.l1p[j]);
            const double d1 = wp - w, d2 = w - wp;
            const bool n1 = signbit(d1) != 0, n2b = signbit(d2) != 0;
            const float sg = n1 ? 1.f : -1.f; // the reference's sign of R(w, w')
            NesItem I;
            dfm::df t = dfm::from_double(w);
            I.wh = t.hi, I.wl = t.lo;
            t = dfm::from_double(wp);
            I.wph = t.hi, I.wpl = t.lo;
            t = dfm::from_double(lw);
            I.lwh = t.hi, I.lwl = t.lo;
            t = dfm::from_double(lwp);
            I.lwph = t.hi, I.lwpl = t.lo;
            I.sefa = sg * neps_exp_f32(d1, n1);
            I.sefb = sg * neps_exp_f32(d2, n2b);
            I.wf   = (float)((r ? L.wx3[i] : L.wx[i]) * L.w2[j]);
            I.pad  = 0.f;
            S.items[k] = I;
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int wid  = threadIdx.x >> 5;
    const int t    = threadIdx.x;
    const int slot = wid / Smem::kWPP, wsub = wid - slot * Smem::kWPP;
    NesPointData& Wd = S.pt[slot];
    uint16_t* qw     = S.q[WIDE ? (wid & 1) : wid];
    // the warps of a point (every thread of them runs the same iterations)
    const auto point_sync = [&]() {
        if (WIDE)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(Smem::kWPP * 32) : "memory");
    };
    const bool nbb  = L.neglect_blocking != 0;
    const bool stim = L.stim != 0;
    constexpr float kBp = (float)k::NepsBPlus, kBm = (float)k::NepsBMinus,
                    kBz = (float)k::NepsBZero;

    for (int64_t qp = (int64_t)blockIdx.x * Smem::kPts + slot; qp < np;
         qp += (int64_t)gridDim.x * Smem::kPts)
    {
        const int64_t p = L.pidx ? L.pidx[p0 + qp] : p0 + qp;
        PointTab* P     = (PointTab*)(scratch + qp * kTabWords);
        const double T = L.eos[1][p], mu_e = L.eos[7][p];
        NepsPoint NP;
        NP.T    = T;
        NP.pre  = k::NepsConst * (T * T);
        NP.eta0 = mu_e / T;
        NP.eta1 = -mu_e / T;
        // range envelope: the occupation of every species far above the FP32
        // normal range at its peak; e^{-Lref} of the e+ integrals finite
        bool ok = isfinite(NP.eta0) && NP.eta0 > -80.;
        if (lane < 4)
        {
            const Distr& d = P->d;
            ok = ok && (d.w_t[lane] == 0. || d.eta_t[lane] > -60.) &&
                 (d.w_f[lane] == 0. || d.beta_f[lane] > 1e-30) && (d.temp_t[lane] > 0.) &&
                 (d.temp_f[lane] > 0.) && isfinite(d.eta_t[lane]) && isfinite(d.beta_f[lane]);
        }
        int flag = __all_sync(0xffffffffu, ok) ? 0 : 2;
        if (flag == 0)
        {
            point_sync(); // the previous point's readers are done
            if (wsub == 0)
            {
                if (lane < 2)
                    Wd.lep[lane] = nes32::make_lepton(lane ? NP.eta1 : NP.eta0);
                else if (lane >= 4 && lane < 16)
                    (&Wd.N.fe[0][0])[lane - 4] = (&P->fe[0][0])[lane - 4];
                else if (lane >= 16 && lane < 18)
                    Wd.N.fd0[lane - 16] = P->fd0[lane - 16];
                else if (lane == 18)
                    Wd.twin = species_twins(P->d);
                else if (lane >= 24 && lane < 28) // x = w = omega / T
                    nu_species(P->d, lane - 24, T, -fx::log(T), &Wd.sp[lane - 24]);
            }
            if (wsub < 2)
            {
#pragma unroll
                for (int kk = 0; kk < 16; ++kk)
                    S.dacc[kk][t] = make_float2(0.f, 0.f);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4)
                    S.mag[k4][t] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            point_sync();
            NP.fd00 = Wd.N.fd0[0];
            NP.fd01 = Wd.N.fd0[1];
            NP.fe0  = Wd.N.fe[0];
            NP.fe1  = Wd.N.fe[1];
            const int nocc = Wd.twin ? 3 : 4;
            // e+ terms scale as e^{-eta_e}: below 1e-13 of the e- terms for eta_e > 30
            const int nlep = NP.eta0 > 30. ? 1 : 2;
            int nq = 0;
            const auto queue_items = [&](int k, unsigned tmk) {
                const unsigned tb = __ballot_sync(0xffffffffu, tmk != 0);
                if (tmk)
                    qw[nq + __popc(tb & ((1u << lane) - 1u))] = (uint16_t)(k | (tmk << 14));
                nq += __popc(tb);
            };
            for (int base = 0; base < nit; base += Smem::kWPP * 32)
            {
                const int k  = base + wsub * 32 + lane;
                unsigned tmk = 0;
                bool any     = false;
                float tm[16];
                if (k < nit)
                {
                    const NesItem I    = S.items[k];
                    const dfm::df W    = {I.wh, I.wl}, WP = {I.wph, I.wpl};
                    const nes32::Geo G = nes32::make_geo(W, WP);
                    // A e^{-Lref}-scaled kernel sum b1 I_1 + b2 I_2 per species
                    // over the leptons: R(nu, nubar) (w w')^2 = sign x c
                    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
                    for (int e = 0; e < nlep; ++e)
                    {
                        const nes32::Lepton& Lp = Wd.lep[e];
                        if (!nes32::above_taylor(G, Lp))
                        {
                            tmk |= 1u << e;
                            continue;
                        }
                        float I1, I2;
                        nes32::lepton_integrals(G, Lp, I1, I2);
                        const float A = Lp.A * I1, B = Lp.A * I2;
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                        {
                            const float bo   = (s < 2) ? kBp : kBm;
                            const bool first = ((s & 1) == 0) != (e == 1); // b1 = bo, b2 = B0
                            c[s] += first ? fmaf(A, bo, B * kBz) : fmaf(A, kBz, B * bo);
                        }
                        any = true;
                    }
                    if (any)
                    {
                        // R(nubar, nu) = -R(nu, nubar)
                        float em1[4], ab1[4], em2[4], ab2[4];
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                        {
                            em1[s] = ab2[s] = -c[s] * I.sefb;
                            ab1[s] = em2[s] = c[s] * I.sefa;
                        }
                        float g[4], gm[4], gb[4], gbm[4];
                        total_nu_q(W, dfm::df{I.lwh, I.lwl}, Wd.sp, nocc, g, gm);
                        total_nu_q(WP, dfm::df{I.lwph, I.lwpl}, Wd.sp, nocc, gb, gbm);
                        nes_terms(stim, nbb, I.wf, I.wh, I.wph, g, gm, gb, gbm, em1, ab1, em2,
                                  ab2, tm);
                    }
                }
                if (!WIDE)
                {
                    if (any)
                        nes_accumulate(S, t, tm);
                    queue_items(k, tmk);
                }
                else
                {
                    // the first two warps add the round's four rows of 64 items in
                    // order, as the two-warp form does
                    S.tmk[t] = (uint8_t)(tmk | (any ? 4u : 0u));
#pragma unroll
                    for (int kk = 0; kk < 16; ++kk)
                        S.tm[kk][t] = tm[kk];
                    __syncthreads();
                    if (wid < 2)
                        for (int v = t; v < Smem::kWPP * 32; v += 64)
                        {
                            const unsigned f = S.tmk[v];
                            if (f & 4u)
                            {
                                float o[16];
#pragma unroll
                                for (int kk = 0; kk < 16; ++kk)
                                    o[kk] = S.tm[kk][v];
                                nes_accumulate(S, t, o);
                            }
                            queue_items(base + v, f & 3u);
                        }
                    __syncthreads();
                }
            }
            __syncwarp();
            // items in the reference's Taylor branches (w or w' below 1e-3 eta,
            // kernel_nes.hpp:82-132), FP64, all lanes busy
            for (int base = 0; base < nq; base += 32)
            {
                const int qi = base + lane;
                if (qi >= nq)
                    continue;
                const unsigned ent = qw[qi];
                const int k        = (int)(ent & 0x3fffu);
                const unsigned tmq = ent >> 14;
                const NesItem I    = S.items[k];
                const double w  = (double)I.wh + (double)I.wl;
                const double wp = (double)I.wph + (double)I.wpl;
                const double x = w > wp ? w : wp, y = w > wp ? wp : w;
                const bool n1 = signbit(wp - w) != 0, n2b = signbit(w - wp) != 0;
                const int sign1 = n1 ? 1 : -1, sign2 = n2b ? 1 : -1;
                const float efa = (float)sign1 * I.sefa, efb = (float)sign1 * I.sefb;
                const float w4  = (float)((w * wp) * (w * wp));
                float em1[4], ab1[4], em2[4], ab2[4];
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    em1[s] = ab1[s] = em2[s] = ab2[s] = 0.f;
#pragma unroll 1
                for (int e = 0; e < 2; ++e)
                {
                    if (!((tmq >> e) & 1u))
                        continue;
                    double t1[4], t2[4];
                    neps_taylor(NP, e, w, wp, x, y, sign1, sign2, t1, t2);
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                    {
                        const float r1 = (float)t1[s] * w4, r2 = (float)t2[s] * w4;
                        em1[s] += -r1 * efb;
                        ab1[s] += r1 * efa;
                        em2[s] += -r2 * efa;
                        ab2[s] += r2 * efb;
                    }
                }
                float g[4], gm[4], gb[4], gbm[4];
                total_nu_q(dfm::df{I.wh, I.wl}, dfm::df{I.lwh, I.lwl}, Wd.sp, nocc, g, gm);
                total_nu_q(dfm::df{I.wph, I.wpl}, dfm::df{I.lwph, I.lwpl}, Wd.sp, nocc, gb, gbm);
                float tm[16];
                nes_terms(stim, nbb, I.wf, I.wh, I.wph, g, gm, gb, gbm, em1, ab1, em2, ab2, tm);
                nes_accumulate(S, t, tm);
            }
            if (wsub < 2)
            {
                double acc[16], mag[16];
#pragma unroll
                for (int kk = 0; kk < 16; ++kk)
                {
                    const float2 a = S.dacc[kk][t];
                    acc[kk]        = (double)a.x + (double)a.y;
                }
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4)
                {
                    const float4 m  = S.mag[k4][t];
                    mag[4 * k4]     = m.x;
                    mag[4 * k4 + 1] = m.y;
                    mag[4 * k4 + 2] = m.z;
                    mag[4 * k4 + 3] = m.w;
                }
                const double ta = warp_sum16(acc, lane), tg = warp_sum16(mag, lane);
                if (!(lane & 1))
                {
                    S.red[slot][wsub][0][sum_index(lane)] = ta;
                    S.red[slot][wsub][1][sum_index(lane)] = tg;
                }
            }
            point_sync();
            if (wsub != 0)
                continue;
            const int idx = sum_index(lane);
            double tot    = S.red[slot][0][0][idx] + S.red[slot][1][0][idx];
            double mtot   = S.red[slot][0][1][idx] + S.red[slot][1][1][idx];
            // terms of both signs (occupation above 1), or NES sums cancelling
            // the pair + brem sums of the same output (those enter the assembly
            // with t2d^2 = hn / 8, times t2d for energy moments) or the beta
            // rates: the point goes to the FP64 pass
            const double unit = NP.pre * ((T * T) * (T * T)) * (idx >= 8 ? T : 1.);
            tot *= unit;
            mtot *= unit;
            const double t2d = k::TempMultiple * T;
            const double other =
                beta_in_sum_unit(P, T, NP.eta0, L.use_abs_em, true, idx) +
                ((L.use_pair || L.use_brem) ? 0.125 * P->s2d[idx] * (idx >= 8 ? t2d : 1.) : 0.);
            if (__any_sync(0xffffffffu, mtot > 0. && mtot > kMaxCancel * fabs(tot + other)))
                flag = 1;
            if (flag == 0 && !(lane & 1)) // else a later launch writes this point's sums
                P->snes[idx] = tot;
        }
        if (wsub == 0 && lane == 0)
        {
            P->neps_fp64 = (double)flag;
            if (flag != 0)
                atomicAdd(&g_grey_mixed[flag], 1ull);
        }
    }
}

// ---------------------------------------------------------------------------
// assembly (m1_opacities.hpp:1172-1294): a CTA takes 32 points, a warp a species of
// them.  Bound by the latency of the record's words and ~12 divisions: with a thread per
// point, all four species in turn, one point took 17 us and now 11, 8,192 points 20 and
// 13.
// ---------------------------------------------------------------------------

// Points whose outputs hold a NaN or Inf (the reference propagates them from
// bad inputs, e.g. GP19 outside its table); read by grey_nonfinite_count.
__device__ unsigned long long g_grey_nonfinite;

template <bool MULTI = false>
__global__ void __launch_bounds__(128)
    grey_final_kernel(const __grid_constant__ OpacityLaunch L0, const GroupArgs GA, int64_t p0,
                      int64_t np, double* __restrict__ scratch, int redo_only)
{
    const OpacityLaunch& L = MULTI ? GA.Ls[blockIdx.z] : L0;
    if (MULTI)
    {
        const GroupChunk& gcz = GA.gc[blockIdx.z];
        p0      = gcz.p0;
        np      = gcz.np;
        scratch = gcz.ws;
    }
    __shared__ uint32_t s_bad[2][3]; // per point: brem, pair sums to redo; not finite
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    if (threadIdx.x < 6)
        s_bad[threadIdx.x / 3][threadIdx.x % 3] = 0u;
    __syncthreads();
    int turn = 0;
    for (int64_t q0 = blockIdx.x * (int64_t)32; q0 < np; q0 += (int64_t)gridDim.x * 32, turn ^= 1)
    {
        const int64_t q     = q0 + lane;
        uint32_t* bad       = s_bad[turn];
        bool nonfinite      = false;
        const bool pcheck   = L.mixed && L.use_pair;
        PointTab* P         = (PointTab*)(scratch + (q < np ? q : q0) * kTabWords);
        const bool run      = q < np && !(redo_only && P->bredo != 1. &&
                                          !(pcheck && pair_mixed(P)->predo == 1.));
        // mixed path: FP32 brem terms whose sum the other reactions cancel
        // (the NES sums of the opposite sign where the occupation exceeds 1)
        // by more than kMaxCancelBrem are recomputed in FP64 (bredo = 1); the
        // same for the FP32 pair integrals beyond kMaxCancelPair (predo = 1)
        const bool check = !redo_only && L.mixed && L.use_brem;
        const bool check_pair = !redo_only && pcheck;
        bool bredo       = false;
        bool predo       = false;
        if (run)
        {
            const int64_t p     = L.pidx ? L.pidx[p0 + q] : p0 + q;
            const double T      = L.eos[1][p];
            const double eta_e  = L.eos[7][p] / T;
            const double t2d    = k::TempMultiple * T;
            const double t2     = t2d * t2d;
            const double tn     = 4. * (k::TempMultiple * T);
            const double hn     = 0.5 * (tn * tn);
            const bool has2d    = L.use_pair || L.use_brem;
            const double sb = s < 2 ? beta_scale(P->fe[s & 1][4], P->fe[s & 1][5], T, eta_e, s) : 0.;
            const double F = k::FourPiHc3, F2 = k::FourPiHc3Sqr, c = k::Clight;
            const double n = L.m1[s][p], J = L.m1[4 + s][p];
            const double s_iso = (n > k::ThresholdN) ? (J / n) : 1.5 * T;
            const double n2d_em = has2d ? P->s2d[s] * t2 : 0.;
            const double n2d_ab = has2d ? P->s2d[4 + s] * t2 : 0.;
            const double e2d_em = has2d ? P->s2d[8 + s] * t2d * t2 : 0.;
            const double e2d_ab = has2d ? P->s2d[12 + s] * t2d * t2 : 0.;
            const double nne_em = L.use_inel ? P->snes[s] * hn : 0.;
            const double nne_ab = L.use_inel ? P->snes[4 + s] * hn : 0.;
            const double ene_em = L.use_inel ? P->snes[8 + s] * hn : 0.;
            const double ene_ab = L.use_inel ? P->snes[12 + s] * hn : 0.;
            const double iso    = L.use_iso ? P->siso[s] * s_iso : 0.;
            double o[5];
            double bne = 0., bje = 0., bna = 0., bja = 0.;
            if (s < 2)
            {
                if (L.use_abs_em)
                {
                    bne = P->sbeta[s] * sb;
                    bje = P->sbeta[2 + s] * sb;
                    bna = P->sbeta[4 + s] * sb;
                    bja = P->sbeta[6 + s] * sb;
                }
                o[0] = F * (F * (n2d_em + nne_em) + bne);
                o[2] = F * (F * (e2d_em + ene_em) + bje);
                o[1] = (n > k::ThresholdN) ? F / (c * n) * (F * (n2d_ab + nne_ab) + bna) : 0.;
                o[3] = (J > k::ThresholdJ) ?
                           ((s == 0 && n == 0.) ? 0. : F / (c * J) * (F * (e2d_ab + ene_ab) + bja)) :
                           0.;
            }
            else
            {
                o[0] = F2 * (n2d_em + nne_em);
                o[2] = F2 * (e2d_em + ene_em);
                o[1] = (n > k::ThresholdN) ?
                           ((s == 3 && n == 0.) ? 0. : F2 / (c * n) * (n2d_ab + nne_ab)) :
                           0.;
                o[3] = (J > k::ThresholdJ) ? F2 / (c * J) * (e2d_ab + ene_ab) : 0.;
            }
            o[4] = (J > k::ThresholdJ) ? F / (c * J) * iso : 0.;
            if (check || check_pair)
            {
                // totals of the four moments before the output factors, and the
                // brem (pair) terms' magnitude in the same units
                const double tot[4] = {F * (n2d_em + nne_em) + bne, F * (n2d_ab + nne_ab) + bna,
                                       F * (e2d_em + ene_em) + bje, F * (e2d_ab + ene_ab) + bja};
#pragma unroll
                for (int m = 0; m < 4; ++m)
                {
                    const double u = F * (m < 2 ? t2 : t2d * t2);
                    if (check)
                        bredo = bredo || u * P->bmag[4 * m + s] > kMaxCancelBrem * fabs(tot[m]);
                    if (check_pair)
                        predo = predo ||
                                u * pair_mixed(P)->pmag[4 * m + s] > kMaxCancelPair * fabs(tot[m]);
                }
            }
#pragma unroll
            for (int qq = 0; qq < 5; ++qq)
            {
                L.out[qq * 4 + s][p] = o[qq];
                nonfinite = nonfinite || !isfinite(o[qq]);
            }
        }
        const uint32_t mb = __ballot_sync(0xffffffffu, bredo), mp = __ballot_sync(0xffffffffu, predo);
        const uint32_t mn = __ballot_sync(0xffffffffu, nonfinite);
        if (lane == 0)
        {
            if (mb)
                atomicOr(&bad[0], mb);
            if (mp)
                atomicOr(&bad[1], mp);
            if (mn)
                atomicOr(&bad[2], mn);
        }
        __syncthreads();
        if (s == 0)
        {
            const uint32_t br = bad[0], pr = bad[1], nf = bad[2];
            const uint32_t mr = __ballot_sync(0xffffffffu, run);
            if (run && !redo_only)
                P->bredo = (br >> lane) & 1u ? 1. : 0.; // also where brem is off: scratch is reused
            if (run && check_pair)
                pair_mixed(P)->predo = (pr >> lane) & 1u ? 1. : 0.;
            if (lane == 0)
            {
                bad[0] = bad[1] = bad[2] = 0u; // for the turn after the next
                if (!redo_only && L.mixed)
                {
                    atomicAdd(&g_grey_mixed[0], (unsigned long long)__popc(mr));
                    if (pr)
                        atomicAdd(&g_grey_mixed[3], (unsigned long long)__popc(pr));
                    if (br)
                        atomicAdd(&g_grey_mixed[4], (unsigned long long)__popc(br));
                }
                if (nf && !redo_only)
                    atomicAdd(&g_grey_nonfinite, (unsigned long long)__popc(nf));
            }
        }
    }
}

// Persistent grid: resident CTAs (occupancy) x num_sms x the launch's
// grid_scale (a tuning knob; 2 by default), capped by the work.
thread_local double g_grid_scale = 1.;

template <class K>
int grid_for(K kernel, int threads, int64_t work, int num_sms)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) !=
            cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    int64_t cap = (int64_t)((double)num_sms * per_sm * g_grid_scale);
    cap = cap < 1 ? 1 : cap;
    return (int)(work < cap ? (work > 0 ? work : 1) : cap);
}

// One step of the phase pipeline.  Single launch (MULTI false): L is the
// launch, points p0 .. p0 + np of it with scratch ws.  Multi-group launch: G
// groups in grid z, their descriptors and chunk shares in GA (device memory);
// L is a host copy whose flags are the union of the groups' (which phases
// run), brem_set the brem variants present (bit i: variant i), np the largest
// share (grid x), p0 and ws unused.
struct Step
{
    OpacityLaunch const* L;
    GroupArgs GA;
    unsigned G;
    unsigned brem_set;
    int64_t p0, np;
    double* ws;
};

// Chunks of fewer points than this many per SM run a point per CTA in the NES
// kernels (both forms add a point's terms in the same order, so its results do
// not depend on the form).  A chip-wide round of the two-warp form is 8 points per
// SM and takes as long for one point as for 1,216; a point per CTA takes time in
// proportion.  FP64, n = 6, 10, 20: a round 80, 162, 553 us; a point per CTA 67, 110,
// 357 us at 600 points, 100, 160, 518 us at 900.  Mixed: a round 95, 135, 346 us; a
// point per CTA 69, 82, 175 us at 300 points (one wave), 115, 144, 314 us at 500.
constexpr int64_t kWide64PerSm = 5, kWideFastPerSm = 2;

// The fast NES pass: 8-warp CTAs with the item table and the per-lane sums in
// dynamic shared memory (two CTAs per SM).
template <bool WIDE, bool MULTI>
cudaError_t launch_nes_fast(const Step& S, cudaStream_t st, int sms)
{
    constexpr int smem = (int)sizeof(NesSmem<WIDE>), kPts = NesSmem<WIDE>::kPts;
    const auto kernel  = grey_nes_fast_kernel<WIDE, MULTI>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               smem);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kNesWarps * 32, smem) !=
            cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    const int64_t work = (S.np + kPts - 1) / kPts;
    int64_t cap        = (int64_t)((double)sms * per_sm * g_grid_scale);
    cap                = cap < 1 ? 1 : cap;
    const int grid     = (int)(work < cap ? (work > 0 ? work : 1) : cap);
    kernel<<<dim3(grid, 1, MULTI ? S.G : 1), kNesWarps * 32, smem, st>>>(*S.L, S.GA, S.p0, S.np,
                                                                         S.ws);
    return cudaGetLastError();
}

template <bool WIDE, bool MULTI>
cudaError_t launch_nes64(const Step& S, cudaStream_t st, int sms, int flagged)
{
    constexpr int NW      = Nes64Smem<WIDE>::kNW;
    constexpr int smem    = (int)sizeof(Nes64Smem<WIDE>);
    const auto kernel     = grey_nes64_kernel<WIDE, MULTI>;
    const cudaError_t e   = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 smem);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, NW * 32, smem) !=
            cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    constexpr int kPts = Nes64Smem<WIDE>::kPts;
    const int64_t work = (S.np + kPts - 1) / kPts;
    int64_t cap        = (int64_t)((double)sms * per_sm * g_grid_scale);
    cap                = cap < 1 ? 1 : cap;
    const int grid     = (int)(work < cap ? (work > 0 ? work : 1) : cap);
    kernel<<<dim3(grid, 1, MULTI ? S.G : 1), NW * 32, smem, st>>>(*S.L, S.GA, S.p0, S.np, S.ws,
                                                                  flagged);
    return cudaGetLastError();
}

// FP64 chunks of at most a point per SM take 256 threads a point in the cell kernels: a
// point's cells in one round instead of four at n = 10.  The row sums stay with the first
// 64 threads, so a point's results do not depend on it.  One point, pair and brem: n = 10
// HR98 64 -> 48 us, n = 20 GP19 124 -> 89; 152 points 68 -> 49, 153 -> 108; 304 points at
// n = 20 157 -> 179.
template <bool MIXED, bool MULTI, int NTW>
void launch_pair_of(const Step& S, cudaStream_t st, int sms, int redo_only)
{
    const auto kernel = grey_pair_kernel<MIXED, MULTI, NTW>;
    kernel<<<dim3(grid_for(kernel, NTW, S.np, sms), 1, MULTI ? S.G : 1), NTW, 0, st>>>(
        *S.L, S.GA, S.p0, S.np, S.ws, redo_only);
}

template <bool MIXED, bool MULTI>
void launch_pair(const Step& S, cudaStream_t st, int sms, int redo_only)
{
    if (!MIXED && !MULTI && S.np <= sms)
        launch_pair_of<MIXED, MULTI, MIXED || MULTI ? kCellThreads : kCellWide>(S, st, sms,
                                                                                redo_only);
    else
        launch_pair_of<MIXED, MULTI, kCellThreads>(S, st, sms, redo_only);
}

template <int IMPL, bool MULTI, int NTW>
void launch_brem64(const Step& S, cudaStream_t st, int sms, int add, bool redo)
{
    const auto k64 = grey_brem_kernel<IMPL, MULTI, NTW>;
    k64<<<dim3(grid_for(k64, NTW, S.np, sms), 1, MULTI ? S.G : 1), NTW, 0, st>>>(
        *S.L, S.GA, S.p0, S.np, S.ws, add, redo ? 1 : 0);
}

// Brem variant IMPL; redo is the FP64 pass over the points the mixed path's
// final kernel marked.
template <int IMPL, bool MULTI>
void launch_brem_impl(const Step& S, cudaStream_t st, int sms, bool mixed, int add, bool redo)
{
    const unsigned gz = MULTI ? S.G : 1;
    phase_mark(kPhBrem, 0, st);
    if (mixed && !redo)
    {
        const auto k32     = grey_brem32_kernel<IMPL, MULTI>;
        const int64_t work = (S.np + kWarps - 1) / kWarps;
        k32<<<dim3(grid_for(k32, kWarps * 32, work, sms), 1, gz), kWarps * 32, 0, st>>>(
            *S.L, S.GA, S.p0, S.np, S.ws, add);
    }
    else if (!MULTI && S.np <= sms)
        launch_brem64<IMPL, MULTI, MULTI ? kCellThreads : kCellWide>(S, st, sms, add, redo);
    else
        launch_brem64<IMPL, MULTI, kCellThreads>(S, st, sms, add, redo);
    phase_mark(kPhBrem, 1, st);
}

// Single launch: the launch's variant; multi-group: one launch per variant
// present (each returns at once for the other variants' groups).
template <bool MULTI>
cudaError_t launch_brem(const Step& S, cudaStream_t st, int sms, bool mixed, int add,
                        bool redo = false)
{
    const unsigned set = MULTI ? S.brem_set : 1u << S.L->brem_impl;
    if (set & 1u)
        launch_brem_impl<0, MULTI>(S, st, sms, mixed, add, redo);
    if (set & 2u)
        launch_brem_impl<1, MULTI>(S, st, sms, mixed, add, redo);
    if (set & 4u)
        launch_brem_impl<2, MULTI>(S, st, sms, mixed, add, redo);
    return cudaGetLastError();
}

template <int IMPL>
cudaError_t launch_small_impl(const Step& S, cudaStream_t st)
{
    constexpr int smem  = (int)sizeof(Nes64Smem<true>);
    const auto kernel   = grey_small_kernel<IMPL>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               smem);
    if (e != cudaSuccess)
        return e;
    phase_mark(kPhNeps, 0, st);
    kernel<<<dim3((unsigned)S.np, S.L->use_inel ? 2 : 1), kCellWide, smem, st>>>(*S.L, S.p0, S.np, S.ws);
    phase_mark(kPhNeps, 1, st);
    return cudaGetLastError();
}

cudaError_t launch_small(const Step& S, cudaStream_t st)
{
    const int impl = S.L->use_brem ? S.L->brem_impl : 1;
    return impl == 0 ? launch_small_impl<0>(S, st)
                     : impl == 1 ? launch_small_impl<1>(S, st) : launch_small_impl<2>(S, st);
}

// FP64 calls of at most this many points per SM take grey_small_kernel for NES beside
// pair or brem, and of at most one for pair and brem alone.  A call's time, each phase by
// itself -> together: one point n = 10 HR98 173 -> 140 us, n = 20 GP19 304 -> 220; 304
// points n = 6 152 -> 143, n = 10 229 -> 211, n = 20 466 -> 415; 456 points 185 -> 180, 280 ->
// 267, 668 -> 611; 608 points 199 -> 208, 313 -> 319, 716 -> 708.
constexpr int64_t kSmallPerSm = 3;

// The phase kernels of one step on stream st: point constants, prelude, pair,
// brem, NES, final, and on the mixed path the FP64 passes over the points the
// final kernel marked, with a second final pass.
template <bool MULTI>
cudaError_t launch_step(const Step& S, cudaStream_t st, int sms)
{
    const OpacityLaunch& L = *S.L;
    const int64_t np       = S.np;
    const unsigned gz      = MULTI ? S.G : 1;
    const bool wide64 = !MULTI && np < kWide64PerSm * sms;
    const bool wide32 = !MULTI && np <= kWideFastPerSm * sms;
    cudaError_t err        = cudaSuccess;
    phase_mark(kPhPrelude, 0, st);
    {
        const int64_t bx = (np + 127) / 128;
        const dim3 pgrid((unsigned)(bx < (int64_t)sms * 4 ? bx : (int64_t)sms * 4), kPointTasks,
                         gz);
        grey_point_kernel<MULTI><<<pgrid, 128, 0, st>>>(L, S.GA, S.p0, np, S.ws);
    }
    phase_mark(kPhPrelude, 1, st);
    phase_mark(kPhPrelude, 0, st);
    grey_prelude_kernel<MULTI>
        <<<dim3(grid_for(grey_prelude_kernel<MULTI>, kPreWarps * 32, np, sms), 1, gz),
           kPreWarps * 32, 0, st>>>(L, S.GA, S.p0, np, S.ws);
    phase_mark(kPhPrelude, 1, st);
    const bool small = !MULTI && !L.mixed &&
                       (L.use_inel ? (L.use_pair || L.use_brem) && np <= kSmallPerSm * sms
                                   : L.use_pair && L.use_brem && np <= sms);
    if (small && (err = launch_small(S, st)) != cudaSuccess)
        return err;
    if (L.use_pair && !small)
    {
        phase_mark(kPhPair, 0, st);
        if (L.mixed)
            launch_pair<true, MULTI>(S, st, sms, 0);
        else
            launch_pair<false, MULTI>(S, st, sms, 0);
        phase_mark(kPhPair, 1, st);
    }
    if (L.use_brem && !small)
    {
        err = launch_brem<MULTI>(S, st, sms, L.mixed != 0, L.use_pair);
        if (err != cudaSuccess)
            return err;
    }
    if (L.use_inel && !small)
    {
        if (L.mixed)
        {
            phase_mark(kPhNeps, 0, st);
            err = wide32 ? launch_nes_fast<true, MULTI>(S, st, sms)
                         : launch_nes_fast<false, MULTI>(S, st, sms);
            if (err != cudaSuccess)
                return err;
            phase_mark(kPhNeps, 1, st);
            phase_mark(kPhNepsAccurate, 0, st);
            grey_nes_list_kernel<MULTI><<<dim3((unsigned)((np + 255) / 256), 1, gz), 256, 0, st>>>(
                L, S.GA, np, S.ws);
            phase_mark(kPhNepsAccurate, 1, st);
            phase_mark(kPhNepsFp64, 0, st);
            if ((err = launch_nes64<true, MULTI>(S, st, sms, 1)) != cudaSuccess)
                return err;
            phase_mark(kPhNepsFp64, 1, st);
        }
        else
        {
            phase_mark(kPhNeps, 0, st);
            err = wide64 ? launch_nes64<true, MULTI>(S, st, sms, 0)
                         : launch_nes64<false, MULTI>(S, st, sms, 0);
            if (err != cudaSuccess)
                return err;
            phase_mark(kPhNeps, 1, st);
        }
    }
    const dim3 fgrid(grid_for(grey_final_kernel<MULTI>, 128, (np + 31) / 32, sms), 1, gz);
    phase_mark(kPhFinal, 0, st);
    grey_final_kernel<MULTI><<<fgrid, 128, 0, st>>>(L, S.GA, S.p0, np, S.ws, 0);
    phase_mark(kPhFinal, 1, st);
    if (L.mixed && (L.use_brem || L.use_pair))
    {
        // points whose FP32 brem or pair sums the other reactions cancel:
        // those parts in FP64, outputs again
        if (L.use_pair)
        {
            phase_mark(kPhPair, 0, st);
            launch_pair<false, MULTI>(S, st, sms, 1);
            phase_mark(kPhPair, 1, st);
        }
        if (L.use_brem && (err = launch_brem<MULTI>(S, st, sms, true, L.use_pair, true)) !=
                              cudaSuccess)
            return err;
        phase_mark(kPhFinal, 0, st);
        grey_final_kernel<MULTI><<<fgrid, 128, 0, st>>>(L, S.GA, S.p0, np, S.ws, 1);
        phase_mark(kPhFinal, 1, st);
    }
    return cudaGetLastError();
}

} // namespace

namespace {

// The mixed path's pair integrals at given (y, z, eta): J_l = e^{ls} j_l with
// J_0 = Psi_0(y, z) / (1 - e^{y+z}), J_1 = Psi_0(z, y) / (1 - e^{y+z})
// (kernel_pair.hpp:16-120), ls = Lref - (y + z).  Zero where the reference
// zeroes Psi (eta - y - z > 200).
__global__ void __launch_bounds__(128)
    pair_j_kernel(const double* __restrict__ y, const double* __restrict__ z,
                  const double* __restrict__ eta, double* __restrict__ j0,
                  double* __restrict__ j1, double* __restrict__ ls, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        pair32::Cell c;
        double lref;
        if (!pair32::make_cell(y[i], z[i], eta[i], c, lref))
        {
            j0[i] = j1[i] = 0.;
            ls[i] = 0.;
            continue;
        }
        double Q0, Q1;
        pair32::cell_integrals(c, Q0, Q1);
        const double yz = y[i] * z[i];
        j0[i] = Q0 / (15. * (yz * yz));
        j1[i] = Q1 / (15. * (yz * yz));
        ls[i] = lref - (y[i] + z[i]);
    }
}

// The mixed path's NES/NPS out-kernel integrals at given (w, w', eta):
// MezzacappaIntOut(w, w', b1, b2) of kernel_nes.hpp:50-78 (the general
// branch, without the Taylor expansions) = e^{ls} (b1 m1 + b2 m2).
__global__ void __launch_bounds__(128)
    nes_m_kernel(const double* __restrict__ w, const double* __restrict__ wp,
                 const double* __restrict__ eta, double* __restrict__ m1,
                 double* __restrict__ m2, double* __restrict__ ls, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
    {
        float I1, I2;
        double lref;
        nes32::lepton_integrals(w[i], wp[i], eta[i], I1, I2, lref);
        const double xy  = w[i] * wp[i];
        const double sgn = w[i] > wp[i] ? 1. : -1.;
        m1[i] = sgn * (double)I1 / (xy * xy);
        m2[i] = sgn * (double)I2 / (xy * xy);
        ls[i] = lref;
    }
}

} // namespace

cudaError_t launch_nes_m(const double* w, const double* wp, const double* eta, double* m1,
                         double* m2, double* ls, int64_t n, cudaStream_t st, int sms)
{
    if (n <= 0)
        return cudaSuccess;
    const int64_t blocks = (n + 127) / 128;
    const int grid       = (int)(blocks < (int64_t)sms * 8 ? blocks : (int64_t)sms * 8);
    phase_mark(kPhAux, 0, st);
    nes_m_kernel<<<grid, 128, 0, st>>>(w, wp, eta, m1, m2, ls, n);
    phase_mark(kPhAux, 1, st);
    return cudaGetLastError();
}

cudaError_t launch_pair_j(const double* y, const double* z, const double* eta, double* j0,
                          double* j1, double* ls, int64_t n, cudaStream_t st, int sms)
{
    if (n <= 0)
        return cudaSuccess;
    const int64_t blocks = (n + 127) / 128;
    const int grid       = (int)(blocks < (int64_t)sms * 8 ? blocks : (int64_t)sms * 8);
    phase_mark(kPhAux, 0, st);
    pair_j_kernel<<<grid, 128, 0, st>>>(y, z, eta, j0, j1, ls, n);
    phase_mark(kPhAux, 1, st);
    return cudaGetLastError();
}

cudaError_t grey_mixed_counts(unsigned long long* counts, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(counts, g_grey_mixed, 5 * sizeof(*counts));
    if (e == cudaSuccess && reset)
    {
        const unsigned long long zero[5] = {0ull, 0ull, 0ull, 0ull, 0ull};
        e = cudaMemcpyToSymbol(g_grey_mixed, zero, sizeof(zero));
    }
    return e;
}

cudaError_t grey_nonfinite_count(unsigned long long* count, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(count, g_grey_nonfinite, sizeof(*count));
    if (e == cudaSuccess && reset)
    {
        const unsigned long long zero = 0ull;
        e = cudaMemcpyToSymbol(g_grey_nonfinite, &zero, sizeof(zero));
    }
    return e;
}

cudaError_t launch_grey_chunks(const OpacityLaunch& L, cudaStream_t st0, cudaStream_t aux, int sms,
                               double* ws0, double* ws1, int64_t chunk, int64_t* k)
{
    if (L.npts <= 0)
        return cudaSuccess;
    if (!ws0 || (aux && !ws1) || chunk < 1 || !k)
        return cudaErrorInvalidValue;
    // default grid: four waves of resident CTAs per phase kernel (per-point
    // work is uneven; later waves fill the tails of earlier ones, and the
    // other stream's kernel the tail of both).  Measured on the 256^3
    // all-reactions slab: 2, 3, 4 waves gave 411k, 417k, 423k points/s mixed
    // (FP64 172k, 174k, 177k); half a wave per stream, so that both streams'
    // kernels stay resident side by side, was 15% slower than 2 waves.
    g_grid_scale = L.grid_scale > 0. ? L.grid_scale : 4.;
    cudaError_t err = cudaSuccess;
    for (int64_t p0 = 0; p0 < L.npts && err == cudaSuccess; p0 += chunk, ++*k)
    {
        const bool odd        = aux != nullptr && (*k & 1);
        const cudaStream_t st = odd ? aux : st0;
        double* const wsk     = odd ? ws1 : ws0;
        const int64_t np      = (L.npts - p0) < chunk ? (L.npts - p0) : chunk;
        const Step S          = {&L, GroupArgs{nullptr, nullptr}, 0u, 0u, p0, np, wsk};
        err                   = launch_step<false>(S, st, sms);
    }
    return err;
}

cudaError_t launch_grey_multi(const OpacityLaunch& U, unsigned brem_set, const GroupArgs& GA,
                              unsigned groups, int64_t np_max, cudaStream_t st, int sms)
{
    if (groups == 0 || np_max <= 0)
        return cudaSuccess;
    if (!GA.Ls || !GA.gc || groups > 65535u)
        return cudaErrorInvalidValue;
    g_grid_scale = U.grid_scale > 0. ? U.grid_scale : 4.;
    const Step S = {&U, GA, groups, brem_set, 0, np_max, nullptr};
    return launch_step<true>(S, st, sms);
}

cudaError_t launch_grey(const OpacityLaunch& L, cudaStream_t st0, int sms, double* ws,
                        int64_t ws_points, cudaStream_t aux)
{
    if (L.npts <= 0)
        return cudaSuccess;
    if (!ws || ws_points < 1)
        return cudaErrorInvalidValue;
    // With an auxiliary stream, consecutive chunks alternate between the
    // caller's stream and aux, each with half of the scratch, so that the
    // FP64-pipe phases (prelude, pair) of one chunk run beside the FP32-pipe
    // NES phase of the other.  The caller's stream waits for aux at the end.
    const bool two      = aux != nullptr && ws_points >= 2 && L.npts > ws_points / 2;
    const int64_t chunk = two ? ws_points / 2 : ws_points;
    cudaEvent_t ev[2]   = {nullptr, nullptr};
    if (two)
    {
        cudaError_t e;
        if ((e = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventRecord(ev[0], st0)) != cudaSuccess ||
            (e = cudaStreamWaitEvent(aux, ev[0], 0)) != cudaSuccess)
            return e;
    }
    int64_t k       = 0;
    cudaError_t err = launch_grey_chunks(L, st0, two ? aux : nullptr, sms, ws,
                                         two ? ws + chunk * kTabWords : nullptr, chunk, &k);
    if (two)
    {
        const cudaError_t e1 = cudaEventRecord(ev[1], aux);
        const cudaError_t e2 = e1 == cudaSuccess ? cudaStreamWaitEvent(st0, ev[1], 0) : e1;
        cudaEventDestroy(ev[0]);
        cudaEventDestroy(ev[1]);
        if (err == cudaSuccess)
            err = e2;
    }
    return err;
}

} // namespace bnsn
