// Spectral opacity kernels (sm_103a), FP64 and mixed precision.
//
// Restates ComputeSpectralOpacities{NotStimulatedAbs,StimulatedAbs} and
// SpectralIntegrand (m1_opacities.hpp:1317-1660).
//
// Phases per chunk of points (the phase split keeps every kernel's code small enough
// for the instruction cache; a single fused kernel spent most cycles waiting on
// instruction fetch):
//   prelude   the constants of each point (distribution parameters, brem, beta and
//             iso constants, Fermi integrals at eta_e) -> chunk scratch;
//   pb        pair + brem sums of every (point, energy) -> records;
//   nes       NES/NPS sums -> records;
//   assemble  beta, iso, the outer factors and the stimulated-absorption
//             correction -> the caller's outputs.
// In FP64 a CTA takes a point in pb and nes (spec_pb64_kernel, spec_nes64_kernel), in
// the mixed path a warp (spec_pb_kernel, spec_nes_kernel).  The antineutrino grid of
// the integral (t x_i, t / x_i with t = 2.182 T for pair/brem, nu x_i, nu / x_i for
// NES) is staged per point or per energy in shared memory.  Each integrand is
// evaluated once per node; the reference evaluates the full integrand once
// per (output, node) (integration.hpp:524-543), which only repeats identical
// values.
//
// MIXED: pb evaluates the pair kernel as the cancellation-free FP32 integral
// of the grey path (bnsn_pair32.cuh) and the brem kernel in FP32 (HR98
// shape, GP19 profiles) with the factor e^{-nu/T} of the emissivity applied
// in FP64 (BRT06 and the GP19 high-T extrapolation stay FP64), and nes rounds its
// FP64 brackets (double-float ones below nu/T = 0.2, in a second launch over those
// energies) to FP32 and multiplies them by FP32 occupation factors formed as
// exponentials of double-float arguments minus a per-energy scale (nes_spec_node), so
// that e^{-(w - w')} g(w') stays in range at any nu/T; per-point data stay FP64 and
// every term is summed in FP64.  Both record an error bound per output: the FP32
// rounding bound (sum|t| over 1.25 for brem, over 2.5 for the pair integrals, over 2
// for NES) plus 1e9 x the components dropped below 2^-120.
// assemble compares the bounds with each output's total.  Where their sum
// exceeds it (terms that cancel), or where a part could not run in FP32
// (bound = inf: occupations outside the FP32 range, NES at nu/T < 0.05), it flags the
// part whose bound exceeds half the total.  Flagged parts are recomputed by the FP64
// kernels over the flagged energies of a point; assemble checks the remaining bounds
// against the totals that now hold the FP64 sums, and a last pass recomputes the outputs
// that fail (pair and brem sums that FP64 NES sums cancel).  (A double-float pass over
// the flagged NES parts before the FP64 one took 2.2 ms of 10.8 per 4,096 points at
// 5% occupancy, and the FP64 kernels are as fast per energy.)
// 4,096 points x 24 energies: FP64 n = 10 HR98 without NES 9.1 -> 1.3 ms, n = 20 GP19
// with NES 17.0 -> 3.9 ms; mixed n = 20 GP19 with NES 12.8 -> 5.5 ms.

#include <algorithm>
#include <type_traits>

#include <cuda_runtime.h>

#include "bnsn_df.cuh"
#include "bnsn_fp32.cuh"
#include "bnsn_fp64.cuh"
#include "bnsn_internal.h"
#include "bnsn_mixed.cuh"
#include "bnsn_pair32.cuh"

namespace bnsn {
namespace {

using namespace fp64;

constexpr int kWarps  = 4;
constexpr int kEChunk = 32; // energies staged per pass

constexpr double kSpecCancelBrem = 1.25;    // sum|t| / |total| of the FP32 brem terms
// same for the FP32 pair integrals: their terms are positive with at most
// 4.1e-7 relative error per cell (bnsn_pair32.cuh), so sum|t| / 2.5 is 1e6 x
// a bound on the error of their sum, the scale of the other bounds
constexpr double kSpecCancelPair = 2.5;
constexpr double kSpecCancelNes  = 2.0;     // same for the NES/NPS terms
constexpr double kSpecNesMinW    = 0.05;    // NES in FP64 below nu/T = 0.05
constexpr double kSpecNesDfW     = 0.2;    // NES brackets in double-float below nu/T = 0.2
constexpr double kSpecFloor      = 7.2e-34; // 1e9 x the denormal floor of a sum

// Per (point, energy) record of the chunk scratch.
struct EnergyRec
{
    double pb[8];   // pair + brem: sum over nodes of w nubar^2 kernel x occupation
    double nes[8];  // NES/NPS: the same
    double bpb[8];  // mixed: error bound of pb[] (inf: recompute in FP64)
    double bnes[8]; // mixed: error bound of nes[]
};

// Kernel modes.
enum SpecMode
{
    kSpecFp64 = 0, // plain path: every energy in FP64
    kSpecMixed,    // mixed path, first pass over every energy
    kSpecRedo,     // FP64 over the flagged energies; assemble re-checks and flags again
    kSpecFinal     // assemble only: the energies flagged twice, no guard
};

// Mixed-path statistics: [0] (point, energy) pairs evaluated, [1] of those
// recomputed in FP64 in any part, [2] pair + brem recomputations, [3] NES
// recomputations.
__device__ unsigned long long g_spec_counts[4];

// (point, energy) pairs whose outputs hold a NaN or Inf.
__device__ unsigned long long g_spec_nonfinite;

// Lane group size for ne energy tasks of M nodes each (power of two <= 32) on a
// number of lanes, minimising rounds x nodes per task.
__host__ __device__ inline int pick_groups(int ne, int M, int lanes)
{
    int best       = 1;
    long best_cost = -1;
    for (int G = 1; G <= 32 && G <= M; G <<= 1)
    {
        const int per_round = lanes / G;
        const long rounds   = (ne + per_round - 1) / per_round;
        const long cost     = rounds * ((M + G - 1) / G);
        if (best_cost < 0 || cost < best_cost)
        {
            best_cost = cost;
            best      = G;
        }
    }
    return best;
}

__device__ __forceinline__ double seg_sum(double v, int G)
{
    for (int o = 1; o < G; o <<= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float seg_sum(float v, int G)
{
    for (int o = 1; o < G; o <<= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// kq-th set bit of m (0-based).
__device__ __forceinline__ int nth_bit(uint64_t m, int kq)
{
    for (int j = 0; j < kq && j < 64; ++j)
        m &= m - 1ull;
    return __ffsll((long long)m) - 1;
}

__device__ __forceinline__ bool same_cf_of(const Distr& d)
{
    const double c0 = d.c_f[0];
    return (d.c_f[1] == c0) && (d.c_f[2] == c0) && (d.c_f[3] == c0);
}

// Occupations of every species at their peaks far inside the FP32 range.
__device__ __forceinline__ bool fp32_envelope(const Distr& d, double eta_e)
{
    bool env = isfinite(eta_e);
#pragma unroll
    for (int s = 0; s < 4; ++s)
        env = env && (d.w_t[s] == 0. || d.eta_t[s] > -60.) &&
              (d.w_f[s] == 0. || d.beta_f[s] > 1e-30) && (d.temp_t[s] > 0.) &&
              (d.temp_f[s] > 0.) && isfinite(d.eta_t[s]) && isfinite(d.beta_f[s]);
    return env;
}

__device__ __forceinline__ uint64_t all_energies(int ne)
{
    return ne >= 64 ? ~0ull : ((1ull << ne) - 1ull);
}

// Energies of point q that an FP64 pass works on (bit e: energy e of the launch).
__device__ __forceinline__ uint64_t energy_mask(const uint64_t* flags, int64_t q, int ne)
{
    return flags ? flags[q] & all_energies(ne) : all_energies(ne);
}

// ---------------------------------------------------------------------------
// prelude: the constants of each point
// ---------------------------------------------------------------------------

// Per point of the chunk scratch.
struct SpecPoint
{
    Distr d;                 // distribution.hpp:51-243
    Occ64 occ[4], occT[4];   // occupations of an energy in MeV, and in units of T
    double fe[2][6], fd0[2]; // F_0..F_5 and FermiDistr(0, 1, .) at +-eta_e
    BetaPoint beta;
    double eta_pp, eta_nn;
    Hr98Point hr;
    Hr98Cell hc;
    double brt06_pre;
    Gp19Point pt;
    Gp19Corners cor[2];
    fp32::Hr98Mixed hm; // mixed path
    NesSpec Z;
    NesDf Q;
    double steep; // T over the lowest temperature of the point
    int twin;     // heavy-lepton neutrinos evolved as one species
    int same_cf, env;
};
static_assert(sizeof(SpecPoint) == 2048, "the documented scratch of a point");

// n doubles of a record into shared memory, by threads t, t + nt, ...
template <class T>
__device__ __forceinline__ void copy_in(T* dst, const T& src, int t, int nt)
{
    static_assert(sizeof(T) % sizeof(double) == 0 && alignof(T) % sizeof(double) == 0,
                  "copied by double words");
    for (int k = t; k < (int)(sizeof(T) / sizeof(double)); k += nt)
        ((double*)dst)[k] = ((const double*)&src)[k];
}

// A CTA takes 32 points, a warp one task of all of them, so every lane works and no
// warp diverges; the second set of tasks needs the first's results.  With the tasks in
// single lanes of the pb and nes kernels, and the beta constants in every lane of
// assemble, they took half the time of 24 energies at n = 10: 4,096 points FP64 HR98
// 1.72 -> 1.27 ms, mixed 2.27 -> 1.97 ms; n = 20 GP19 with NES mixed 5.87 -> 5.5 ms.
constexpr int kPreTasks = 15;

__global__ void __launch_bounds__(kPreTasks * 32)
    spec_prelude_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0, int64_t np,
                        SpecPoint* __restrict__ pts)
{
    const int64_t q  = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const int task   = threadIdx.x >> 5;
    const bool in    = q < np;
    const int64_t p  = p0 + (in ? q : 0);
    SpecPoint& P     = pts[in ? q : 0];
    const bool hr98  = L.use_brem && L.brem_impl == 0;
    const bool prof  = L.use_brem && L.brem_impl == 2 && L.gp19.d3 <= kGp19MaxW;
    const double T   = L.eos[1][p], mu_e = L.eos[7][p], nbar = L.eos[0][p];
    const double yp = L.eos[3][p], yn = L.eos[4][p], eta = mu_e / T;
    if (in)
    {
        if (task < 4)
        {
            Distr& d    = P.d;
            const int s = task;
            if (L.has_distr)
                for (int k = 0; k < 7; ++k)
                    (&d.w_t[0])[k * 4 + s] = L.distr[k * 4 + s][p];
            else
                distr_species(L.m1[s][p], L.m1[4 + s][p], L.m1[8 + s][p], L.gamma36, &d.w_t[s],
                              &d.temp_t[s], &d.eta_t[s], &d.w_f[s], &d.temp_f[s], &d.c_f[s],
                              &d.beta_f[s]);
        }
        else if (task < 7 && hr98)
            P.hr.ch[task - 4] = hr98_channel(nbar, yn, yp, T, task - 4);
        else if (task == 7 && hr98)
            hr98_point_common(nbar, T, L.use_medium != 0, &P.hr);
        else if (task == 8 && L.use_brem && L.brem_impl == 1)
            P.brt06_pre = brt06_point(nbar, T, yn, yp);
        else if (task == 8 && prof)
            gp19_point(gp19_table(L), nbar, L.eos[2][p], T, &P.pt);
        else if (task == 9 && L.use_abs_em)
            P.beta = beta_point(nbar, T, yp, yn, L.eos[5][p], L.eos[6][p], mu_e, L.eos[9][p],
                                L.eos[10][p], L.use_dU, L.use_dm_eff, L.use_WM_ab, L.use_decay);
        else if (task == 10)
        {
            P.eta_pp = L.use_iso ? eta_nn_sc(nbar, T, yp) : 0.;
            P.eta_nn = L.use_iso ? eta_nn_sc(nbar, T, yn) : 0.;
        }
        else if (task == 11 || task == 12)
        {
            const double e = task == 12 ? -eta : eta;
            fdi_orders<0, 5>(e, P.fe[task - 11]);
            P.fd0[task - 11] = fermi_distr(0., 1., e);
        }
        else if (task >= 13 && L.mixed && L.use_inel)
        {
            const int e  = task - 13;
            P.Q.eta[e]   = dfm::from_double(e ? -eta : eta);
            dfm::fdi_raw15(P.Q.eta[e], P.Q.reta[e], 1, &dfm::kFdiTab);
        }
    }
    __syncthreads();
    if (!in)
        return;
    const Distr& d = P.d;
    if (task < 4)
    {
        occ64_from(d, task, 1., &P.occ[task]);
        occ64_from(d, task, T, &P.occT[task]);
        if (L.mixed)
            nes_spec_species(d, task, &P.Z);
    }
    else if (task < 8 && hr98)
        hr98_cell_from(P.hr, task - 4, &P.hc);
    else if (task >= 8 && task < 12 && hr98 && L.mixed)
        fp32::hr98_mixed_part(P.hr, task - 8, &P.hm);
    else if (task >= 12 && task < 14 && prof)
    {
        const int k = task - 12;
        if (k == 0 || P.pt.regime >= 2)
            gp19_profile_corners(gp19_table(L), P.pt.nbp, P.pt.yep, P.pt.pT[k], &P.cor[k]);
    }
    else if (task == 14)
    {
        P.twin    = species_twins(d);
        P.same_cf = same_cf_of(d);
        P.env     = fp32_envelope(d, eta);
        if (L.mixed)
            nes_spec_masks(d, &P.Z);
        double t = T;
        for (int s = 0; s < 4; ++s)
            t = fmin(t, fmin(d.temp_t[s], d.temp_f[s]));
        P.steep = T / t;
    }
}

// ---------------------------------------------------------------------------
// pb: pair annihilation + NN bremsstrahlung
// ---------------------------------------------------------------------------
struct PbWarp
{
    Distr d;
    Hr98Point hr;
    double nb[kMaxM], zb[kMaxM]; // nubar and nubar / T
    double gb[kMaxM][4];
    Gp19Point gp;
    Gp19Corners gc[2];
    double gpp[2][kGp19MaxW];
};

struct PbWarpMixed
{
    fp32::Hr98Mixed hm;
    float yeh[kEChunk], yel[kEChunk]; // nu / T as hi + lo
    float ybh[kMaxM], ybl[kMaxM];     // nubar / T as hi + lo
    double ehy[kEChunk], dny[kEChunk]; // pair: e^{y - cy}, e^{-y} of the energies
    double ehz[kMaxM], dnz[kMaxM];     // the same of the nodes
    float gb32[kMaxM][4], gbm32[kMaxM][4];
    float gp32[2][kGp19MaxW];
};

struct PbShared
{
    double x[kMaxQ], B1[kMaxM];
    dfm::df B1d[kMaxM]; // mixed: weights as double-float
    double lw[kGp19MaxW], wax[kGp19MaxW], iw[kGp19MaxW];
    float lwf[kGp19MaxW], idl[kGp19MaxW];
    PbWarp w[kWarps];
    PbWarpMixed m[kWarps];
};

// GP19 kernel of one node from the per-point profiles in FP64.
__device__ __forceinline__ void gp19_profile_node(const Gp19Point& gp,
                                                  const double (*gpp)[kGp19MaxW],
                                                  const double* lw, int d3, double wmin,
                                                  double wmax, double nu, double nub, double* be,
                                                  double* ba)
{
    double w = nu + nub;
    w        = w > wmax ? wmax : (w < wmin ? wmin : w);
    double tw;
    const int l     = bracket_sorted<double>(log(w), lw, d3, &tw);
    const double v0 = gpp[0][l] * (1. - tw) + gpp[0][l + 1] * tw;
    const double v1 = gp.regime >= 2 ? gpp[1][l] * (1. - tw) + gpp[1][l + 1] * tw : 0.;
    gp19_cell(gp, v0, v1, w, nu + nub, be, ba);
}

// Pair + brem in FP64: every energy, or (flags) the ones the mixed path's checks
// flagged.  A CTA takes a point: the node and energy tables (Fermi integrals,
// occupations times weights) over its threads, then the (energy, node) cells'
// absorption kernels (pair, both orders of Psi, and brem; emission is e^{-(nu +
// nubar)/T} of it) into shared memory, then a thread per (energy, output) sums its
// row.  Bound by the FP64 pipe and the integer work of the fixed-point exponentials.
// With a warp per point whose lanes split the nodes of an energy and carried eight
// sums each, the node tables were 4x as much shared memory a resident warp, a third
// of the lanes idled at n = 10, and a flagged energy held a whole warp of a nearly
// empty grid.  Energies below kPairLowEnergy T take a second pass of their own
// (rational Fermi integrals, the reference's order of sums).
constexpr int kPbCells = 32 * 21; // cells of a pass: 32 energies at M = 20, 16 at M = 40
template <int IMPL>
struct Pb64Brem
{
};
template <>
struct Pb64Brem<0>
{
    Hr98Cell hc;
};
template <>
struct Pb64Brem<2>
{
    Gp19Point pt;
    Gp19Corners gc[2];
    double p[2][kGp19MaxW];
    Gp19Axis axis;
};

template <int IMPL>
struct Pb64Smem
{
    double x[kMaxQ];
    Occ64 occ[4];
    double fe[2];                              // F_3, F_4 at eta_e
    double nb[kMaxM], z[kMaxM], iz2[kMaxM], dnz[kMaxM]; // nubar, z = nubar / T, 1 / z^2, e^{-z}
    double vE[4][kMaxM], vA[4][kMaxM];         // w nubar^2 (1 - g) e^{-z}, w nubar^2 g
    double fm[kMaxM][5], fp[kMaxM][5];         // node tables at eta -+ z
    int eid[kEChunk];
    double nu[kEChunk], y[kEChunk], iy2[kEChunk], dny[kEChunk];
    int far[kEChunk];                          // a node with (nu + nubar) / T > 700
    double em[kEChunk][5], ep[kEChunk][5];     // energy tables at eta -+ y
    double K[3][kPbCells];                     // pair Psi(y, z), Psi(z, y), brem
    Pb64Brem<IMPL> X;
};

// A cell with x = (nu + nubar) / T > 700 from the pair kernel's sum of Psi and the brem
// absorption kernel.  There the reference clamps e^x at e^700, its emission kernel
// rounds in the denormal range and the pair absorption kernel is e^700 times that,
// so both are formed in its order.  BRT06's emission kernel is not clamped.
template <int IMPL>
__device__ __noinline__ double pb64_far(double psi, double Kbrem, double T, double x, int ab)
{
    const double ex = safe_exp(x);
    const double em = 0.5 * (psi * (k::PairPhi * (T * T) / (1. - ex)));
    return ab ? ex * em + Kbrem : em + (IMPL == 1 ? brt06_emission(Kbrem, 0.5 * x) : Kbrem * safe_exp(-x));
}

template <int IMPL>
__global__ void __launch_bounds__(kWarps * 32, 4)
    spec_pb64_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0,
                     const SpecPoint* __restrict__ pts, EnergyRec* __restrict__ rec,
                     const uint64_t* __restrict__ flags)
{
    constexpr int NT = kWarps * 32;
    const int64_t q  = blockIdx.x;
    const int n = L.n1, M = 2 * n, ne = L.n_energies, tid = threadIdx.x;
    const uint64_t emask = energy_mask(flags, q, ne);
    if (emask == 0ull)
        return;
    __shared__ Pb64Smem<IMPL> S;
    const SpecPoint& P = pts[q];
    const int64_t p    = p0 + q;
    const double T = L.eos[1][p], eta = L.eos[7][p] / T;
    const bool pair = L.use_pair != 0, brem = L.use_brem != 0;
    const bool nbb  = L.neglect_blocking != 0;
    const Gp19Table G19 = gp19_table(L);
    const bool prof     = IMPL == 2 && brem && G19.d3 <= kGp19MaxW;
    if (tid < n)
        S.x[tid] = L.x1[tid];
    if (tid >= 32 && tid < 64)
        copy_in(&S.occ, P.occ, tid - 32, 32);
    if constexpr (IMPL == 0)
        if (brem && tid >= 64 && tid < 96)
            copy_in(&S.X.hc, P.hc, tid - 64, 32);
    if constexpr (IMPL == 2)
        if (prof)
        {
            if (tid >= 64 && tid < 96)
            {
                copy_in(&S.X.pt, P.pt, tid - 64, 32);
                copy_in(&S.X.gc, P.cor, tid - 64, 32);
            }
            if (tid >= 96)
                for (int k = tid - 96; k < G19.d3; k += 32)
                    gp19_axis_entry(S.X.axis, G19.logw, G19.d3, k);
        }
    __syncthreads();
    // antineutrino grid (m1_opacities.hpp:1542)
    const double ts   = k::TempMultiple * T;
    const bool common = S.occ[0].cf == k::CF && S.occ[1].cf == k::CF && S.occ[2].cf == k::CF &&
                        S.occ[3].cf == k::CF;
    for (int t = tid; t < 4 * M; t += NT)
    {
        const int a = t >> 2, s = t & 3;
        const double nub = a < n ? ts * S.x[a] : ts / S.x[a - n];
        const double g   = occ64_one(S.occ[s], nub, fx::pow(nub, common ? k::CF : S.occ[s].cf));
        const double z = nub / T, dz = safe_exp(-z), wn = L.B1[a] * (nub * nub);
        // species s ^ 1 is the partner of s
        S.vE[s ^ 1][a] = (nbb ? wn : wn * (1. - g)) * dz;
        S.vA[s ^ 1][a] = wn * g;
        if (s == 0)
        {
            S.nb[a]  = nub;
            S.z[a]   = z;
            S.iz2[a] = 1. / (z * z);
            S.dnz[a] = dz;
        }
    }
    if constexpr (IMPL == 2)
        if (prof)
        {
            const int np19 = S.X.pt.regime >= 2 ? 2 : 1;
            for (int e = tid; e < np19 * G19.d3; e += NT)
            {
                const int pr = e / G19.d3, l = e - pr * G19.d3;
                S.X.p[pr][l] = gp19_profile_eval(G19, S.X.gc[pr], l);
            }
        }
    uint64_t low = 0ull;
    if (pair)
        for (int e = 0; e < ne; ++e)
            low |= (uint64_t)(L.energies[e] < kPairLowEnergy * T) << e;
    const int Ms = M + 1, nc_max = kPbCells / Ms < kEChunk ? kPbCells / Ms : kEChunk;
    const double scp = -0.5 * k::PairPhi * (T * T);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass)
    {
        const uint64_t mask = emask & (pass ? low : ~low);
        const int nt        = __popcll(mask);
        if (nt == 0)
            continue;
        const int chunks = (nt + nc_max - 1) / nc_max, per = (nt + chunks - 1) / chunks;
        __syncthreads(); // the node tables' readers are done
        if (pair)
            for (int t = tid; t < 2 * M + 1; t += NT)
            {
                if (t == 2 * M)
                {
                    if (pass)
                        fdi_rational<3, 4>(eta, S.fe);
                    else
                    {
                        S.fe[0] = P.fe[0][3];
                        S.fe[1] = P.fe[0][4];
                    }
                    continue;
                }
                const int a = t >> 1;
                const double arg = t & 1 ? eta + S.z[a] : eta - S.z[a];
                double* o        = t & 1 ? S.fp[a] : S.fm[a];
                if (pass)
                    fdi_rational<1, 5>(arg, o);
                else
                {
                    double f[5];
                    fdi_orders<1, 5>(arg, f);
                    pair_scale(f, o);
                }
            }
#pragma unroll 1
        for (int k0 = 0; k0 < nt; k0 += per)
        {
            const int nc = nt - k0 < per ? nt - k0 : per;
            __syncthreads(); // the last chunk's readers are done
            for (int t = tid; t < 2 * nc; t += NT)
            {
                const int c = t >> 1, e = nth_bit(mask, k0 + c);
                const double nu = L.energies[e], y = nu / T;
                if ((t & 1) == 0)
                {
                    S.eid[c] = e;
                    S.nu[c]  = nu;
                    S.y[c]   = y;
                    S.iy2[c] = 1. / (y * y);
                    S.dny[c] = safe_exp(-y);
                    S.far[c] = 0;
                }
                if (pair)
                {
                    const double arg = t & 1 ? eta + y : eta - y;
                    double* o        = t & 1 ? S.ep[c] : S.em[c];
                    if (pass)
                        fdi_rational<1, 5>(arg, o);
                    else
                    {
                        double f[5];
                        fdi_orders<1, 5>(arg, f);
                        pair_scale(f, o);
                    }
                }
            }
            __syncthreads();
            const double f40 = 40. * S.fe[0], f20 = 20. * S.fe[1];
            for (int t = tid; t < nc * M; t += NT)
            {
                const int c = t / M, a = t - c * M;
                const double y = S.y[c], z = S.z[a], ex = S.dny[c] * S.dnz[a];
                const bool far = y + z > k::ExpUpp;
                if (far)
                    S.far[c] = 1;
                double q0 = 0., q1 = 0., Kb = 0.;
                if (pair)
                {
                    double f = far ? 1. : scp * fx::rcp(1. - ex); // far: Psi itself
                    if (pass)
                        pair_psi_low(eta, y, z, S.em[c], S.ep[c], S.fm[a], S.fp[a], S.fe[0],
                                     S.fe[1], &q0, &q1);
                    else if (!(eta - y - z > 200.))
                    {
                        pair_psi_scaled(S.em[c], S.ep[c], S.fm[a], S.fp[a], eta, y, z, f40, f20,
                                        &q0, &q1);
                        f *= (S.iy2[c] * S.iz2[a]) * (1. / 15.);
                    }
                    q0 *= f;
                    q1 *= f;
                }
                if (brem)
                {
                    if constexpr (IMPL == 0)
                    {
                        double b;
                        if (S.X.hc.fast && y > 1e-6 && y < 4e4)
                            Kb = hr98_absorption(S.X.hc, y + z, ex);
                        else
                            hr98_kernel(P.hr, S.nu[c], S.nb[a], &b, &Kb);
                    }
                    else if constexpr (IMPL == 1)
                        Kb = P.brt06_pre * brt06_shape(0.5 * (y + z));
                    else
                    {
                        double b;
                        if (prof)
                            Kb = gp19_profile_absorption(
                                S.X.pt, S.X.p, S.X.axis, G19.d3,
                                fmax(fmin(S.nu[c] + S.nb[a], G19.w[G19.d3 - 1]), G19.w[0]));
                        else
                            gp19_kernel(G19, L.eos[0][p], L.eos[2][p], T, S.nu[c], S.nb[a], &b, &Kb);
                    }
                }
                const int o = c * Ms + a;
                S.K[0][o] = q0;
                S.K[1][o] = q1;
                S.K[2][o] = Kb;
            }
            __syncthreads();
            for (int t = tid; t < 8 * nc; t += NT)
            {
                const int c = t >> 3, s = t & 3, ab = (t >> 2) & 1;
                constexpr double e0 = k::PairA1e * k::PairA1e, e1 = k::PairA2e * k::PairA2e;
                constexpr double x0 = k::PairA1x * k::PairA1x, x1 = k::PairA2x * k::PairA2x;
                const double c0 = s < 2 ? e0 : x0, c1 = s < 2 ? e1 : x1;
                const double* K0 = S.K[s & 1] + c * Ms;
                const double* K1 = S.K[1 - (s & 1)] + c * Ms;
                const double* Kb = S.K[2] + c * Ms;
                const double* v  = ab ? S.vA[s] : S.vE[s];
                double acc       = 0.;
                if (S.far[c])
                    for (int a = 0; a < M; ++a)
                    {
                        const double x = S.y[c] + S.z[a], Kp = fma(c0, K0[a], c1 * K1[a]);
                        const double wn = L.B1[a], nb2 = S.nb[a] * S.nb[a];
                        // a weight that underflows (T < 1e-10) belongs to a term that does
                        const double den = fmax((ab ? 1. : S.dnz[a]) * (wn * nb2), 2.3e-308);
                        const double g   = !ab && nbb ? 1. : v[a] / den;
                        const double K = x > k::ExpUpp ? pb64_far<IMPL>(Kp, Kb[a], T, x, ab)
                                                       : (Kp + Kb[a]) * (ab ? 1. : safe_exp(-x));
                        acc += wn * (nb2 * (K * g));
                    }
                else
                    for (int a = 0; a < M; ++a)
                        acc = fma(fma(c0, K0[a], fma(c1, K1[a], Kb[a])), v[a], acc);
                EnergyRec& E       = rec[q * ne + S.eid[c]];
                E.pb[4 * ab + s]  = ab || S.far[c] ? acc : acc * S.dny[c];
                E.bpb[4 * ab + s] = 0.;
            }
        }
    }
}

// Launches of fewer points than this many per SM share a point's energies between warps. A
// pair cell is a chain of ~10 us, and a warp's slowest lane sets its time: 16 points x 40
// energies, pair alone, n = 20: a warp per point 1.57 ms, shared 0.74; 16 x 24 with HR98
// 0.81 -> 0.43. 304 points x 24, n = 10, pair: 0.48 -> 0.41; 608: no difference. With 8 per SM
// 456 points x 40 with HR98 at n = 20 take 2.38 ms instead of 2.22 (every warp makes the node
// tables).
constexpr int64_t kPbWarpsPerSm = 4;

// Pair + brem of the mixed path: a warp takes a point, or (SHARED) every parts-th energy of
// one; an energy's sums do not depend on it.  (One kernel for both, with parts = 1, was 2%
// slower on large calls.)
template <bool SHARED>
__global__ void __launch_bounds__(kWarps * 32)
    spec_pb_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0, int64_t np,
                   const SpecPoint* __restrict__ pts, EnergyRec* __restrict__ rec, int G, int parts)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    PbShared& S         = *reinterpret_cast<PbShared*>(s_raw);
    const Gp19Table G19 = gp19_table(L);
    const bool prof   = L.use_brem && L.brem_impl == 2 && G19.d3 <= kGp19MaxW;
    const double wmin = prof ? G19.w[0] : 0., wmax = prof ? G19.w[G19.d3 - 1] : 0.;
    for (int k = threadIdx.x; k < kMaxQ; k += blockDim.x)
        S.x[k] = L.x1[k];
    for (int k = threadIdx.x; k < kMaxM; k += blockDim.x)
    {
        S.B1[k]  = L.B1[k];
        S.B1d[k] = dfm::from_double(L.B1[k]);
    }
    if (prof)
        for (int k = threadIdx.x; k < G19.d3; k += blockDim.x)
        {
            S.lw[k]  = G19.logw[k];
            S.lwf[k] = (float)G19.logw[k];
            S.wax[k] = G19.w[k];
            S.iw[k]  = 1. / G19.w[k];
            S.idl[k] = k + 1 < G19.d3 ? (float)(1. / (G19.logw[k + 1] - G19.logw[k])) : 0.f;
        }
    __syncthreads();

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    PbWarp& W      = S.w[wid];
    PbWarpMixed& X = S.m[wid];
    const int n = L.n1, M = 2 * n, ne = L.n_energies;
    const bool nbb      = L.neglect_blocking != 0;
    const int64_t nwarp = (int64_t)gridDim.x * kWarps;
    const int grp = lane % G, per_round = 32 / G;

    const int64_t tasks = SHARED ? np * parts : np;
    for (int64_t t = (int64_t)blockIdx.x * kWarps + wid; t < tasks; t += nwarp)
    {
        const int64_t q     = SHARED ? t / parts : t;
        const int part      = SHARED ? (int)(t - q * parts) : 0;
        const int64_t p     = p0 + q;
        const double T = L.eos[1][p], eta_e = L.eos[7][p] / T;
        EnergyRec* R       = rec + q * ne;
        const SpecPoint& P = pts[q];
        __syncwarp();
        copy_in(&W.d, P.d, lane, 32);
        if (L.use_brem && L.brem_impl == 0)
        {
            copy_in(&W.hr, P.hr, lane, 32);
            copy_in(&X.hm, P.hm, lane, 32);
        }
        if (prof)
        {
            copy_in(&W.gp, P.pt, lane, 32);
            copy_in(&W.gc, P.cor, lane, 32);
            __syncwarp();
            const int np19 = (W.gp.regime >= 2) ? 2 : 1;
            for (int e = lane; e < np19 * G19.d3; e += 32)
            {
                const int pr = e / G19.d3, l = e - pr * G19.d3;
                const double v = gp19_profile_eval(G19, W.gc[pr], l);
                W.gpp[pr][l] = v;
                X.gp32[pr][l] = (float)v;
            }
        }
        __syncwarp();
        const bool same_cf = P.same_cf != 0;
        // mixed pair: eta and the point's factor (Phi T^2 / 2) T^4 / 15
        const dfm::df ETA = dfm::from_double(eta_e);
        const double T2   = T * T;
        const double scq  = 0.5 * k::PairPhi * T2 * (T2 * T2) / 15.;
        // shares of |eta| in e^{Lref} = e^{y - cy} e^{z - cz}, used where y + z <= |eta|: halves,
        // or beyond 1,400, where those leave the double range, 300 on the node's side (z < 640)
        const double aeta = fabs(eta_e), cz = aeta <= 1400. ? 0.5 * aeta : 300., cy = aeta - cz;
        // antineutrino grid of the pair/brem integral (m1_opacities.hpp:1542)
        const double ts = k::TempMultiple * T;
        for (int a = lane; a < M; a += 32)
        {
            const int i     = a < n ? a : a - n;
            const double nu = a < n ? ts * S.x[i] : ts / S.x[i];
            W.nb[a]         = nu;
            W.zb[a]         = nu / T;
            total_nu_f4(nu, W.d, same_cf, W.gb[a]);
            const dfm::df yd = dfm::from_double(nu / T);
            X.ybh[a] = yd.hi;
            X.ybl[a] = yd.lo;
            if (L.use_pair)
            {
                X.ehz[a] = fx::exp(W.zb[a] - cz);
                X.dnz[a] = fx::exp(-W.zb[a]);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s)
            {
                X.gb32[a][s]  = (float)W.gb[a][s];
                X.gbm32[a][s] = (float)(1. - W.gb[a][s]);
            }
        }
        // FP32 brem for HR98 and the GP19 profiles (not the high-T
        // extrapolation) inside the FP32 range envelope
        bool b32  = false;
        double sb = 0.;
        float thr = 0.f, lt2 = 0.f;
        if (L.use_brem)
        {
            b32 = (L.brem_impl == 0 || (prof && W.gp.regime != 3 && W.gp.regime != 5)) &&
                  P.env;
            if (L.brem_impl == 0)
                sb = (T * T) * X.hm.outer;
            else if (prof)
            {
                sb  = (T * T) * (3. * W.gp.C);
                thr = (float)(1e-30 / W.gp.C);
                lt2 = (float)log2(T * 0.5);
            }
        }
        // brem in FP64 here when FP32 does not apply, except the full-table GP19
        // kernel (w axis longer than the profiles hold), left to the FP64 redo
        const bool skip = L.use_brem && !b32 && L.brem_impl == 2 && !prof;

        for (int e0 = 0; e0 < ne; e0 += kEChunk)
        {
            const int nec     = (ne - e0) < kEChunk ? (ne - e0) : kEChunk;
            __syncwarp();
            for (int c = lane; c < nec; c += 32)
            {
                const double y   = L.energies[e0 + c] / T;
                const dfm::df yd = dfm::from_double(y);
                X.yeh[c] = yd.hi;
                X.yel[c] = yd.lo;
                if (L.use_pair)
                {
                    X.ehy[c] = fx::exp(y - cy);
                    X.dny[c] = fx::exp(-y);
                }
            }
            __syncwarp();
            // the part's energies: e = part, part + parts, ...
            const int first = SHARED ? (part + parts - e0 % parts) % parts : 0;
            const int own   = !SHARED ? nec : first < nec ? (nec - first + parts - 1) / parts : 0;
            for (int r0 = 0; r0 < own; r0 += per_round)
            {
                const bool act  = r0 + lane / G < own;
                const int k     = act ? r0 + lane / G : 0;
                const int c     = SHARED ? (act ? k * parts + first : 0) : k;
                const double nu = act ? L.energies[e0 + c] : 1.;
                const double w  = nu / T;
                double acc[8];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    acc[kk] = 0.;
                float gl[8]; // sum|t| / 1.25 + 1e9 x dropped
                double gp[8]; // sum|t| of the FP32 pair terms
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                {
                    gl[kk] = 0.f;
                    gp[kk] = 0.;
                }
                const double sbe = sb * fx::exp(-w); // brem emission carries e^{-nu/T}
                const double inu2 = 1. / (nu * nu);
                if (act && !skip)
                {
                    for (int a = grp; a < M; a += G)
                    {
                        const double wa  = S.B1[a];
                        const double nub = W.nb[a];
                        const double* gb = W.gb[a];
                        double be = 0., ba = 0.;
                        if (L.use_brem && !b32)
                        {
                            if (L.brem_impl == 0)
                                hr98_kernel(W.hr, nu, nub, &be, &ba);
                            else if (L.brem_impl == 1)
                                brt06_kernel(P.brt06_pre, T, nu, nub, &be, &ba);
                            else if (prof)
                                gp19_profile_node(W.gp, W.gpp, S.lw, G19.d3, wmin, wmax, nu,
                                                  nub, &be, &ba);
                            const double nb2 = nub * nub;
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                            {
                                const int ps    = s ^ 1;
                                const double bf = nbb ? 1. : 1. - gb[ps];
                                acc[s] += wa * (nb2 * (be * bf));
                                acc[4 + s] += wa * (nb2 * (ba * gb[ps]));
                            }
                        }
                        if (L.use_pair)
                        {
                            // FP32 pair integral: (em, ab) (nu nubar)^2, positive
                            double qe[4], qa[4];
                            pair32::kernel_q(dfm::df{X.yeh[c], X.yel[c]},
                                             dfm::df{X.ybh[a], X.ybl[a]}, X.ehy[c], X.ehz[a],
                                             X.dny[c], X.dnz[a], ETA, scq, qe, qa);
                            const double wq = wa * inu2;
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                            {
                                const int ps    = s ^ 1;
                                const double bf = nbb ? 1. : 1. - gb[ps];
                                const double te = wq * (qe[s] * bf);
                                const double ta = wq * (qa[s] * gb[ps]);
                                acc[s] += te;
                                acc[4 + s] += ta;
                                gp[s] += fabs(te);
                                gp[4 + s] += fabs(ta);
                            }
                        }
                        if (b32)
                        {
                            // kernel shape at x = (nu + nubar) / T (hi + lo)
                            const dfm::df xs = dfm::add(dfm::df{X.yeh[c], X.yel[c]},
                                                        dfm::df{X.ybh[a], X.ybl[a]});
                            float kab;
                            bool slow = false;
                            if (L.brem_impl == 0)
                                kab = fp32::hr98_shape(X.hm, xs.hi, xs.lo);
                            else
                            {
                                double wv = nu + nub;
                                wv        = wv > wmax ? wmax : (wv < wmin ? wmin : wv);
                                float tw;
                                const int l = gp19_bracket32(wv, S.lwf, S.wax, S.iw, S.idl,
                                                             G19.d3, &tw);
                                const float v0 =
                                    X.gp32[0][l] + tw * (X.gp32[0][l + 1] - X.gp32[0][l]);
                                if (W.gp.regime <= 1)
                                    kab = v0;
                                else
                                {
                                    const float v1 =
                                        X.gp32[1][l] + tw * (X.gp32[1][l + 1] - X.gp32[1][l]);
                                    kab = v0 * exp2f(log2f(v1 / v0) * lt2);
                                    // regime 2 clips at 1e-30: exact FP64 node
                                    slow = W.gp.regime == 2 &&
                                           (v0 < thr || v1 < thr || kab < thr);
                                }
                                kab = fabsf(kab);
                            }
                            // e^{-nubar/T}; below 2^-120 the term is dropped
                            const bool far = X.ybh[a] > -kNesDropArg;
                            float kem = far ? 0.f : kab * (expf(-X.ybh[a]) * (1.f - X.ybl[a]));
                            if (slow)
                            {
                                double em, abv;
                                gp19_profile_node(W.gp, W.gpp, S.lw, G19.d3, wmin, wmax, nu,
                                                  nub, &em, &abv);
                                kab = (float)(abv / (3. * W.gp.C));
                                kem = (float)(em * exp(w) / (3. * W.gp.C));
                            }
                            // w nubar^2 / T^2 rounded once from double-float factors
                            const dfm::df yb  = {X.ybh[a], X.ybl[a]};
                            const dfm::df wyd = dfm::mul(S.B1d[a], dfm::mul(yb, yb));
                            const float wy2   = wyd.hi + wyd.lo;
#pragma unroll
                            for (int s = 0; s < 4; ++s)
                            {
                                const int ps = s ^ 1;
                                float bf32   = nbb ? 1.f : X.gbm32[a][ps];
                                float g32    = X.gb32[a][ps];
                                float dre    = far ? wy2 * kab * kNesDrop : 0.f;
                                float dra    = 0.f;
                                if (fabsf(bf32) < kNesDrop)
                                {
                                    dre += wy2 * kem * kNesDrop;
                                    bf32 = 0.f;
                                }
                                if (g32 < kNesDrop)
                                {
                                    dra += wy2 * kab * kNesDrop;
                                    g32 = 0.f;
                                }
                                const float te = wy2 * (kem * bf32);
                                const float ta = wy2 * (kab * g32);
                                acc[s]     = fma(sbe, (double)te, acc[s]);
                                acc[4 + s] = fma(sb, (double)ta, acc[4 + s]);
                                gl[s] += fabsf(te) * (float)(1. / kSpecCancelBrem) + 1e9f * dre;
                                gl[4 + s] +=
                                    fabsf(ta) * (float)(1. / kSpecCancelBrem) + 1e9f * dra;
                            }
                        }
                    }
                }
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                {
                    acc[kk] = seg_sum(acc[kk], G);
                    gl[kk]  = seg_sum(gl[kk], G);
                    if (L.use_pair)
                        gp[kk] = seg_sum(gp[kk], G);
                }
                if (act && grp == 0)
                {
                    EnergyRec& E = R[e0 + c];
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                    {
                        E.pb[kk]  = acc[kk];
                        E.bpb[kk] = skip ? INFINITY
                                         : (b32 ? (kk < 4 ? sbe : sb) * ((double)gl[kk] + kSpecFloor)
                                                : 0.) +
                                               gp[kk] * (1. / kSpecCancelPair);
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// nes: inelastic neutrino-electron / -positron scattering
// ---------------------------------------------------------------------------
struct NesWarp
{
    double fe[2][6];
    double fw[kEChunk][2][5]; // Fermi integrals at eta_e - nu/T (nes_spec_node)
    NesSpec Z;
    NesDf Q;
    dfm::df lnu[kEChunk];
};

struct NesShared
{
    double x[kMaxQ], xinv[kMaxQ], B1[kMaxM];
    dfm::df lxd[kMaxQ];
    dfm::FdiTab ftab;
    NesWarp w[kWarps];
};

// NES/NPS in FP64: every energy, or (flags) the ones the mixed path's checks
// flagged.  A CTA takes a point; groups of G consecutive lanes take an energy and
// split its nodes.  An energy w = nu/T enters its nodes (w x_i, w / x_i) only
// through one bracket per lepton (nes_bracket): the couplings of the four species,
// the factors 1 / (1 - e) of NEPSExpFunc and the occupations follow from it, and the
// node's weight nubar^2 cancels the bracket's 1 / w'^2.  Bound by the FP64 pipe beside
// the integer work of its Fermi integrals and exponentials.
struct Nes64Smem
{
    double x[kMaxQ], xinv[kMaxQ], xc[kMaxQ], xci[kMaxQ]; // nodes, x^0.6 and inverses
    double m[kMaxM];                                     // 24 x weight
    Occ64 occ[4];
    double fe[2][6], fd0[2];
    double w[kEChunk], wc[kEChunk];     // nu/T and its 0.6th power
    double fw[kEChunk][2][5];           // phi_1..phi_5 at eta_e - nu/T
    int eid[kEChunk];
};

// 1 - e^{-d} for e = e^{-d}, d >= 0: by its series below d = 1/4 (2^-53 relative).
__device__ __forceinline__ double one_minus_exp(double d, double e)
{
    if (d >= 0.25)
        return 1. - e;
    double t = 1. / 479001600.;
    t = fma(t, -d, 1. / 39916800.);
    t = fma(t, -d, 1. / 3628800.);
    t = fma(t, -d, 1. / 362880.);
    t = fma(t, -d, 1. / 40320.);
    t = fma(t, -d, 1. / 5040.);
    t = fma(t, -d, 1. / 720.);
    t = fma(t, -d, 1. / 120.);
    t = fma(t, -d, 1. / 24.);
    t = fma(t, -d, 1. / 6.);
    t = fma(t, -d, 0.5);
    return fma(d * d, -t, d);
}

// Emission term of species s at a node of an energy so high that everything it emits
// is next to 0: the reference clamps its exponentials at e^-700 and the products
// round in the denormal range, so they are taken in its order.  A0, B0
// and A1, B1: the brackets of e- and e+; m = 24 x weight; f: the NEPSExpFunc factor.
__device__ __noinline__ double nes64_far(int s, double A0, double B0, double A1, double B1,
                                         double w, double wp, double T, double m, double f,
                                         double g)
{
    const double P = w * wp, nub = wp * T;
    const double h = 24. * k::NepsConst * (T * T) / (P * P);
    const double b = s < 2 ? k::NepsBPlus : k::NepsBMinus, z = k::NepsBZero;
    const double r0 = s & 1 ? z * A0 + b * B0 : b * A0 + z * B0;
    const double r1 = s & 1 ? b * A1 + z * B1 : z * A1 + b * B1;
    const double em = __dadd_rn(__dmul_rn(h * r0, f), __dmul_rn(h * r1, f));
    return m * (1. / 24.) * (nub * nub * __dmul_rn(em, g));
}

__global__ void __launch_bounds__(kWarps * 32, 4)
    spec_nes64_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0,
                      const SpecPoint* __restrict__ pts, EnergyRec* __restrict__ rec,
                      const uint64_t* __restrict__ flags)
{
    constexpr int NT = kWarps * 32;
    const int64_t q  = blockIdx.x;
    const int n = L.n1, M = 2 * n, ne = L.n_energies, tid = threadIdx.x;
    const uint64_t emask = energy_mask(flags, q, ne);
    if (emask == 0ull)
        return;
    __shared__ Nes64Smem S;
    const int64_t p  = p0 + q;
    const double T   = L.eos[1][p], eta_e = L.eos[7][p] / T;
    const bool nbb   = L.neglect_blocking != 0;
    const double sc  = k::NepsConst * (T * T) * (T * T);
    if (tid < n)
    {
        const double x = L.x1[tid], xi = 1. / x;
        S.x[tid]    = x;
        S.xinv[tid] = xi;
        S.xc[tid]   = fx::pow(x, k::CF);
        S.xci[tid]  = fx::pow(xi, k::CF);
    }
    if (tid >= 64 && tid < 64 + M)
        S.m[tid - 64] = 24. * L.B1[tid - 64];
    const SpecPoint& P = pts[q];
    if (tid >= 32 && tid < 64)
    {
        copy_in(&S.occ, P.occT, tid - 32, 32);
        copy_in(&S.fe, P.fe, tid - 32, 32);
        copy_in(&S.fd0, P.fd0, tid - 32, 32);
    }
    const int nt = __popcll(emask);
    const int G  = pick_groups(nt < kEChunk ? nt : kEChunk, M, NT);
    const int grp = tid % G, per_round = NT / G;
    const int chunks = (nt + kEChunk - 1) / kEChunk, per = (nt + chunks - 1) / chunks;
#pragma unroll 1
    for (int k0 = 0; k0 < nt; k0 += per)
    {
        const int nc = nt - k0 < per ? nt - k0 : per;
        __syncthreads(); // the last chunk's readers are done
        for (int t = tid; t < 2 * nc; t += NT)
        {
            const int c = t >> 1, e = nth_bit(emask, k0 + c);
            const double w = L.energies[e] / T;
            if ((t & 1) == 0)
            {
                S.eid[c] = e;
                S.w[c]   = w;
                S.wc[c]  = fx::pow(w, k::CF);
            }
            fx::fd_orders<1, 5, true>((t & 1 ? -eta_e : eta_e) - w, S.fw[c][t & 1]);
        }
        __syncthreads();
        const Occ64* occ  = S.occ;
        const bool common = occ[0].cf == k::CF && occ[1].cf == k::CF && occ[2].cf == k::CF &&
                            occ[3].cf == k::CF;
        const int nocc = P.twin ? 3 : 4;
#pragma unroll 1
        for (int r0 = 0; r0 < nc; r0 += per_round)
        {
            const bool act = r0 + tid / G < nc;
            const int c    = act ? r0 + tid / G : 0;
            const double w = S.w[c];
            const bool tiny = !(w * P.steep < 500.); // e^-500: emission near the denormals
            double acc[8];
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                acc[kk] = 0.;
#pragma unroll 1
            for (int a = act ? grp : M; a < M; a += G)
            {
                const bool down = a < n; // w' < w: the neutrino loses energy
                const int i     = down ? a : a - n;
                const double wp = w * (down ? S.x[i] : S.xinv[i]);
                const double x = down ? w : wp, y = down ? wp : w, dl = x - y;
                double U = 0., V = 0.; // A of e- + B of e+, B of e- + A of e+
                double A = 0., B = 0.; // at the end those of e+
#pragma unroll 1
                for (int e = 0; e < 2; ++e)
                {
                    const double eta = e ? -eta_e : eta_e;
                    const double* fe = S.fe[e];
                    if (y > eta * 1e-3)
                    {
                        double f[5];
                        const double* g = S.fw[c][e];
                        fx::fd_orders<1, 5, true>(eta - wp, f);
                        nes_bracket(eta, x, y, dl, down ? g : f, down ? f : g, fe, &A, &B);
                    }
                    else
                        nes_bracket_taylor(eta, x, y, dl, fe, S.fd0[e], &A, &B);
                    U += e ? B : A;
                    V += e ? A : B;
                }
                constexpr double bp = k::NepsBPlus, bm = k::NepsBMinus, bz = k::NepsBZero;
                const double zU = bz * U, zV = bz * V;
                const double r[4] = {fma(bp, U, zV), fma(bp, V, zU), fma(bm, U, zV),
                                     fma(bm, V, zU)};
                // NEPSExpFunc: e / (1 - e) up and 1 / (1 - e) down in energy
                const double ex = safe_exp(-dl);
                const double kb = S.m[a] * fx::rcp(one_minus_exp(dl, ex) + (dl == 0.));
                const double ka = kb * ex;
                const double ke = down ? ka : kb, kk = down ? kb : ka;
                const double pc = common ? S.wc[c] * (down ? S.xc[i] : S.xci[i]) : 0.;
                double g = 0.;
#pragma unroll
                for (int s = 0; s < 4; ++s)
                {
                    if (s < nocc)
                        g = occ64_one(occ[s], wp, common ? pc : fx::pow(wp, occ[s].cf));
                    if (tiny)
                        acc[s] += nes64_far(s, U - B, V - A, A, B, w, wp, T, S.m[a],
                                            ke / S.m[a], g) * (w * w / sc);
                    else
                        acc[s] = fma(ke * r[s], g, acc[s]);
                    acc[4 + s] = fma(kk * r[s], nbb ? 1. : 1. - g, acc[4 + s]);
                }
            }
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
                acc[kk] = seg_sum(acc[kk], G);
            if (act && grp == 0)
            {
                EnergyRec& E   = rec[q * ne + S.eid[c]];
                const double f = sc * fx::rcp(w * w);
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                {
                    E.nes[kk]  = f * acc[kk];
                    E.bnes[kk] = 0.;
                }
            }
        }
    }
}

// NES/NPS of the mixed path.
template <bool LOW>
__global__ void __launch_bounds__(kWarps * 32, 4)
    spec_nes_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0, int64_t np,
                    const SpecPoint* __restrict__ pts, EnergyRec* __restrict__ rec)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    NesShared& S = *reinterpret_cast<NesShared*>(s_raw);
    for (int k = threadIdx.x; k < kMaxQ; k += blockDim.x)
    {
        S.x[k]    = L.x1[k];
        S.xinv[k] = 1. / L.x1[k];
        S.lxd[k]  = dfm::from_double(L.lx1[k]);
    }
    for (int k = threadIdx.x; k < kMaxM; k += blockDim.x)
        S.B1[k] = L.B1[k];
    for (int k = threadIdx.x; LOW && k < (int)(sizeof(dfm::FdiTab) / sizeof(float)); k += blockDim.x)
        ((float*)&S.ftab)[k] = ((const float*)&dfm::kFdiTab)[k];
    __syncthreads();

    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    NesWarp& W     = S.w[wid];
    const int n = L.n1, M = 2 * n, ne = L.n_energies;
    const bool nbb      = L.neglect_blocking != 0;
    const int64_t nwarp = (int64_t)gridDim.x * kWarps;

    for (int64_t q = (int64_t)blockIdx.x * kWarps + wid; q < np; q += nwarp)
    {
        const int64_t p     = p0 + q;
        const double T = L.eos[1][p], mu_e = L.eos[7][p];
        const double eta_e = mu_e / T, invT = 1. / T;
        EnergyRec* R       = rec + q * ne;
        if (LOW)
        {
            bool any = false;
            for (int e = lane; e < ne; e += 32)
                any = any || !(L.energies[e] / T >= kSpecNesDfW);
            if (!__any_sync(0xffffffffu, any))
                continue;
        }
        __syncwarp();
        const SpecPoint& P = pts[q];
        copy_in(&W.fe, P.fe, lane, 32);
        copy_in(&W.Z, P.Z, lane, 32);
        if (LOW)
            copy_in(&W.Q, P.Q, lane, 32);
        __syncwarp();
        NepsPoint NP;
        NP.T    = T;
        NP.pre  = k::NepsConst * (T * T);
        NP.eta0 = eta_e;
        NP.eta1 = -eta_e;
        NP.fd00 = P.fd0[0];
        NP.fd01 = P.fd0[1];
        NP.fe0  = W.fe[0];
        NP.fe1  = W.fe[1];
        const bool m32  = P.env != 0;
        const double sn = (T * T) * NP.pre;

        for (int e0 = 0; e0 < ne; e0 += kEChunk)
        {
            const int nec     = (ne - e0) < kEChunk ? (ne - e0) : kEChunk;
            __syncwarp();
            // this kernel's energies of the chunk; LOW: those below kSpecNesDfW, and
            // the ones left to the FP64 pass (bound = inf)
            const double wl = lane < nec ? L.energies[e0 + lane] / T : 0.;
            const bool runl = m32 && wl >= kSpecNesMinW, lowl = !(wl >= kSpecNesDfW);
            const uint32_t mask = __ballot_sync(0xffffffffu, runl && lowl == LOW);
            if (lane < nec)
            {
                W.lnu[lane] = dfm::from_double(log(L.energies[e0 + lane]));
                if (!runl && lowl == LOW)
                {
                    EnergyRec& E = R[e0 + lane];
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                    {
                        E.nes[kk]  = 0.;
                        E.bnes[kk] = INFINITY;
                    }
                }
            }
            for (int t = lane; t < 2 * nec; t += 32)
            {
                const int c = t >> 1, e = t & 1;
                if (!((mask >> c) & 1u))
                    continue;
                const double a = (e ? NP.eta1 : NP.eta0) - L.energies[e0 + c] / T;
                if (LOW)
                    dfm::fdi_raw15(dfm::from_double(a), (dfm::df*)W.fw[c][e], 1, &S.ftab);
                else
                    fx::fd_orders<1, 5, true>(a, W.fw[c][e]);
            }
            __syncwarp();
            // G lanes an energy
            const int nt = __popc(mask), G = pick_groups(nt, M, 32), grp = lane & (G - 1);
            for (int r0 = 0; r0 * 32 < nt * G; ++r0)
            {
                const int kq    = (r0 * 32 + lane) / G;
                const bool act  = kq < nt;
                const int c     = act ? nth_bit(mask, kq) : 0;
                const double nu = act ? L.energies[e0 + c] : 1.;
                const double w  = nu / T;
                double acc[8];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    acc[kk] = 0.;
                float gl[8];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                    gl[kk] = 0.f;
                float sig[2] = {0.f, 0.f};
                // scale of this energy: group-wide maximum of the lanes' scans
                nes_spec_scan(W.Z, (float)w, (float)nu, W.lnu[c].hi, S.x, S.lxd, n,
                              act ? grp : M, G, nbb, sig);
                for (int o = 1; o < G; o <<= 1)
                {
                    sig[0] = fmaxf(sig[0], __shfl_xor_sync(0xffffffffu, sig[0], o));
                    sig[1] = fmaxf(sig[1], __shfl_xor_sync(0xffffffffu, sig[1], o));
                }
                sig[0] = isfinite(sig[0]) ? sig[0] : 0.f;
                sig[1] = isfinite(sig[1]) ? sig[1] : 0.f;
                const double sne = sn * fx::exp((double)sig[0]);
                const double sna = sn * fx::exp((double)sig[1]);
                const dfm::df Wd = dfm::from_double(w);
                if (act)
                {
                    for (int a = grp; a < M; a += G)
                    {
                        const int i = a < n ? a : a - n;
                        // nubar/T and log nubar without divisions
                        const double nub = nu * (a < n ? S.x[i] : S.xinv[i]);
                        const double wp  = nub * invT;
                        const dfm::df NB = dfm::from_double(nub), WPd = dfm::from_double(wp);
                        const dfm::df LB =
                            dfm::add(W.lnu[c], a < n ? S.lxd[i] : dfm::neg(S.lxd[i]));
                        float te[4], ta[4], de[4], da[4];
                        nes_spec_node(NP, W.Z, w, wp, Wd, WPd, NB, LB, (float)S.B1[a], sig[0],
                                      sig[1], nbb, W.fw[c], LOW ? &W.Q : nullptr, &S.ftab, te, ta, de, da);
#pragma unroll
                        for (int s = 0; s < 4; ++s)
                        {
                            acc[s]     = fma(sne, (double)te[s], acc[s]);
                            acc[4 + s] = fma(sna, (double)ta[s], acc[4 + s]);
                            gl[s] += fabsf(te[s]) * (float)(1. / kSpecCancelNes) + 1e9f * de[s];
                            gl[4 + s] +=
                                fabsf(ta[s]) * (float)(1. / kSpecCancelNes) + 1e9f * da[s];
                        }
                    }
                }
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                {
                    acc[kk] = seg_sum(acc[kk], G);
                    gl[kk]  = seg_sum(gl[kk], G);
                }
                if (act && grp == 0)
                {
                    EnergyRec& E = R[e0 + c];
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                    {
                        E.nes[kk]  = acc[kk];
                        E.bnes[kk] = (kk < 4 ? sne : sna) * ((double)gl[kk] + kSpecFloor);
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// assemble (m1_opacities.hpp:1571-1660)
// ---------------------------------------------------------------------------
// Only the second check marks records; in the other modes they are read-only.
template <int MODE>
using AssembleRec = std::conditional_t<MODE == kSpecRedo, EnergyRec, const EnergyRec>;

template <int MODE>
__global__ void __launch_bounds__(kWarps * 32)
    spec_assemble_kernel(const __grid_constant__ OpacityLaunch L, int64_t p0, int64_t np,
                         const SpecPoint* __restrict__ pts, AssembleRec<MODE>* __restrict__ rec,
                         uint64_t* __restrict__ fl_pb, uint64_t* __restrict__ fl_nes)
{
    constexpr bool GUARD = MODE == kSpecMixed || MODE == kSpecRedo;
    __shared__ Distr s_d[kWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Distr& D       = s_d[wid];
    const int ne   = L.n_energies;
    const bool pb  = L.use_pair || L.use_brem;
    const int64_t nwarp = (int64_t)gridDim.x * kWarps;
    for (int64_t q = (int64_t)blockIdx.x * kWarps + wid; q < np; q += nwarp)
    {
        uint64_t emask = all_energies(ne);
        if (MODE == kSpecRedo || MODE == kSpecFinal)
        {
            emask &= fl_pb[q] | fl_nes[q];
            if (emask == 0ull)
                continue;
        }
        const int64_t p    = p0 + q;
        const double T     = L.eos[1][p];
        const SpecPoint& P = pts[q];
        __syncwarp();
        copy_in(&D, P.d, lane, 32);
        __syncwarp();
        const bool same_cf  = P.same_cf != 0;
        const BetaPoint& bp = P.beta;
        const double eta_pp = P.eta_pp, eta_nn = P.eta_nn;
        const double ts = k::TempMultiple * T;
        uint64_t bad_pb = 0ull, bad_nes = 0ull;
        for (int e0 = 0; e0 < ne; e0 += 32)
        {
            const int e    = e0 + lane;
            const bool act = e < ne && ((emask >> e) & 1ull);
            bool fpb = false, fnes = false;
            if (act)
            {
                const double nu    = L.energies[e];
                const EnergyRec& E = rec[q * ne + e];
                double b_ab[4] = {0., 0., 0., 0.}, b_em[4] = {0., 0., 0., 0.};
                if (L.use_abs_em)
                {
                    beta_rates(bp, nu, 0, &b_ab[0], &b_em[0]);
                    beta_rates(bp, nu, 1, &b_ab[1], &b_em[1]);
                }
                const double F = k::FourPiHc3, c = k::Clight;
                double ip[8], in[8];
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)
                {
                    ip[kk] = pb ? ts * E.pb[kk] : 0.;
                    in[kk] = L.use_inel ? nu * E.nes[kk] : 0.;
                }
                if constexpr (MODE == kSpecFinal)
                    if (((fl_pb[q] >> e) & 1ull) && !((fl_nes[q] >> e) & 1ull))
                        for (int kk = 0; kk < 8; ++kk)
                            if (!isnan(E.bnes[kk])) // not flagged by the second check
                                ip[kk] = ts * E.bnes[kk];
                if (GUARD)
                {
                    // FP32 error bounds against each output's total
                    uint32_t pb_of = 0u; // outputs whose pair + brem part is flagged
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                    {
                        const int s      = kk & 3;
                        const double tot = (kk < 4 ? b_em[s] : b_ab[s]) + F * (ip[kk] + in[kk]);
                        const double bb  = pb ? F * ts * E.bpb[kk] : 0.;
                        const double bn  = L.use_inel ? F * nu * E.bnes[kk] : 0.;
                        const double at  = fabs(tot);
                        if (!(bb + bn <= at))
                        {
                            // the parts above half of a finite total (at least
                            // one is); both when neither is (or the total is
                            // not finite).  A bound is ~1e6 x the part's actual
                            // error, so redoing one part hardly moves the total
                            // and the kept part stays below half of it.
                            bool xp = bb > 0., xn = bn > 0.;
                            const bool hp = xp && !(bb <= 0.5 * at);
                            const bool hn = xn && !(bn <= 0.5 * at);
                            if (hp || hn)
                            {
                                xp = hp;
                                xn = hn;
                            }
                            pb_of |= (uint32_t)xp << kk;
                            fnes = fnes || xn;
                        }
                    }
                    fpb = pb_of != 0u;
                    // the outputs that pass the second check keep their sums: set aside
                    // (NaN where flagged) in words that are free once NES has passed
                    if constexpr (MODE == kSpecRedo)
                        if (fpb && !fnes)
                            for (int kk = 0; kk < 8; ++kk)
                                rec[q * ne + e].bnes[kk] =
                                    (pb_of >> kk) & 1u ? __longlong_as_double(0x7ff8000000000000LL)
                                                       : E.pb[kk];
                }
                if (!fpb && !fnes)
                {
                    bool nonfinite = false;
                    double ge[4];
                    total_nu_f4(nu, D, same_cf, ge);
                    const double iso =
                        L.use_iso ? iso_scatt_leg0(nu, eta_pp, eta_nn, L.use_WM_sc != 0) : 0.;
                    const int64_t o = p * L.e_stride + L.e_offset + e;
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                    {
                        const double g = ge[s];
                        double j  = b_em[s] + F * (ip[s] + in[s]);
                        double ka = (b_ab[s] + F * (ip[4 + s] + in[4 + s])) / c;
                        double js = 4. * k::Pi * (nu * nu) * g * iso;
                        double ks = 4. * k::Pi * (nu * nu) * (1. - g) * iso / c;
                        if (L.stim)
                        {
                            ka = j / c + ka;
                            ks = js / c + ks;
                        }
                        L.sout[s][o]      = j;
                        L.sout[4 + s][o]  = ka;
                        L.sout[8 + s][o]  = js;
                        L.sout[12 + s][o] = ks;
                        nonfinite = nonfinite || !isfinite(j) || !isfinite(ka) ||
                                    !isfinite(js) || !isfinite(ks);
                    }
                    if (nonfinite)
                        atomicAdd(&g_spec_nonfinite, 1ull);
                }
            }
            if (GUARD)
            {
                bad_pb |= (uint64_t)__ballot_sync(0xffffffffu, fpb) << e0;
                bad_nes |= (uint64_t)__ballot_sync(0xffffffffu, fnes) << e0;
            }
        }
        if (GUARD && lane == 0)
        {
            fl_pb[q]  = bad_pb;
            fl_nes[q] = bad_nes;
            if (MODE == kSpecMixed)
            {
                atomicAdd(&g_spec_counts[0], (unsigned long long)ne);
                atomicAdd(&g_spec_counts[1], (unsigned long long)__popcll(bad_pb | bad_nes));
            }
            atomicAdd(&g_spec_counts[2], (unsigned long long)__popcll(bad_pb));
            atomicAdd(&g_spec_counts[3], (unsigned long long)__popcll(bad_nes));
        }
    }
}

// Dynamic shared memory opt-in (once per kernel) and a persistent grid of two
// waves of resident CTAs, capped by the work.
template <class K>
cudaError_t grid_of(K kernel, size_t smem, bool* attr_set, int num_sms, int64_t warps_needed,
                    int* grid)
{
    cudaError_t err;
    if (!*attr_set)
    {
        if ((err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem)) != cudaSuccess)
            return err;
        *attr_set = true;
    }
    int per_sm = 0;
    if ((err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kWarps * 32, smem)) !=
        cudaSuccess)
        return err;
    per_sm             = per_sm < 1 ? 1 : per_sm;
    const int64_t need = (warps_needed + kWarps - 1) / kWarps;
    const int64_t cap  = (int64_t)num_sms * per_sm * 2;
    *grid              = (int)(need < cap ? need : cap);
    return cudaSuccess;
}

template <bool SHARED>
cudaError_t launch_pb_form(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                           EnergyRec* rec, int G, int parts, cudaStream_t st, int sms)
{
    static bool attr  = false;
    const size_t smem = sizeof(PbShared);
    int grid          = 0;
    cudaError_t err   = grid_of(spec_pb_kernel<SHARED>, smem, &attr, sms, np * parts, &grid);
    if (err != cudaSuccess || grid == 0)
        return err;
    phase_mark(kPhSpectral, 0, st);
    spec_pb_kernel<SHARED><<<grid, kWarps * 32, smem, st>>>(L, p0, np, pts, rec, G, parts);
    phase_mark(kPhSpectral, 1, st);
    return cudaGetLastError();
}

cudaError_t launch_pb_mixed(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                            EnergyRec* rec, int G, cudaStream_t st, int sms)
{
    const int64_t parts = std::min<int64_t>(sms * kPbWarpsPerSm / np, L.n_energies);
    return parts > 1 ? launch_pb_form<true>(L, p0, np, pts, rec, G, (int)parts, st, sms)
                     : launch_pb_form<false>(L, p0, np, pts, rec, G, 1, st, sms);
}

cudaError_t launch_nes_mixed(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                             EnergyRec* rec, cudaStream_t st, int sms)
{
    static bool attr[2] = {false, false};
    const size_t smem   = sizeof(NesShared);
    int grid = 0, low = 0;
    cudaError_t err = grid_of(spec_nes_kernel<false>, smem, &attr[0], sms, np, &grid);
    if (err == cudaSuccess)
        err = grid_of(spec_nes_kernel<true>, smem, &attr[1], sms, np, &low);
    if (err != cudaSuccess || grid == 0)
        return err;
    phase_mark(kPhSpectral, 0, st);
    spec_nes_kernel<false><<<grid, kWarps * 32, smem, st>>>(L, p0, np, pts, rec);
    phase_mark(kPhSpectral, 1, st);
    phase_mark(kPhSpectral, 0, st);
    spec_nes_kernel<true><<<low, kWarps * 32, smem, st>>>(L, p0, np, pts, rec);
    phase_mark(kPhSpectral, 1, st);
    return cudaGetLastError();
}

// FP64 passes: every energy (flags null) or the flagged ones.
cudaError_t launch_pb64(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                        EnergyRec* rec, const uint64_t* flags, cudaStream_t st)
{
    phase_mark(kPhSpectral, 0, st);
    const int impl = L.use_brem ? L.brem_impl : 1;
    if (impl == 0)
        spec_pb64_kernel<0><<<(int)np, kWarps * 32, 0, st>>>(L, p0, pts, rec, flags);
    else if (impl == 1)
        spec_pb64_kernel<1><<<(int)np, kWarps * 32, 0, st>>>(L, p0, pts, rec, flags);
    else
        spec_pb64_kernel<2><<<(int)np, kWarps * 32, 0, st>>>(L, p0, pts, rec, flags);
    phase_mark(kPhSpectral, 1, st);
    return cudaGetLastError();
}

cudaError_t launch_nes64(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                         EnergyRec* rec, const uint64_t* flags, cudaStream_t st)
{
    phase_mark(kPhSpectral, 0, st);
    spec_nes64_kernel<<<(int)np, kWarps * 32, 0, st>>>(L, p0, pts, rec, flags);
    phase_mark(kPhSpectral, 1, st);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_assemble(const OpacityLaunch& L, int64_t p0, int64_t np, const SpecPoint* pts,
                            EnergyRec* rec, uint64_t* fl_pb, uint64_t* fl_nes,
                            cudaStream_t st, int sms)
{
    static bool attr = false;
    int grid         = 0;
    cudaError_t err  = grid_of(spec_assemble_kernel<MODE>, 0, &attr, sms, np, &grid);
    if (err != cudaSuccess || grid == 0)
        return err;
    phase_mark(kPhSpectral, 0, st);
    spec_assemble_kernel<MODE><<<grid, kWarps * 32, 0, st>>>(L, p0, np, pts, rec, fl_pb, fl_nes);
    phase_mark(kPhSpectral, 1, st);
    return cudaGetLastError();
}

} // namespace

int64_t spectral_chunk_points(int n_energies)
{
    const int64_t ne = n_energies < 1 ? 1 : n_energies;
    const int64_t c  = std::min(kSpecChunkRecords / ne,
                                kSpecChunkBytes / (int64_t)spectral_scratch_bytes(1, (int)ne));
    return c < 32 ? 32 : c;
}

size_t spectral_scratch_bytes(int64_t chunk_points, int n_energies)
{
    return (size_t)chunk_points *
           (sizeof(SpecPoint) + 2 * sizeof(uint64_t) + (size_t)n_energies * sizeof(EnergyRec));
}

cudaError_t spectral_mixed_counts(unsigned long long* counts, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(counts, g_spec_counts, sizeof(g_spec_counts));
    if (e == cudaSuccess && reset)
    {
        const unsigned long long zero[4] = {0ull, 0ull, 0ull, 0ull};
        e = cudaMemcpyToSymbol(g_spec_counts, zero, sizeof(zero));
    }
    return e;
}

cudaError_t spectral_nonfinite_count(unsigned long long* count, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(count, g_spec_nonfinite, sizeof(*count));
    if (e == cudaSuccess && reset)
    {
        const unsigned long long zero = 0ull;
        e = cudaMemcpyToSymbol(g_spec_nonfinite, &zero, sizeof(zero));
    }
    return e;
}

cudaError_t launch_spectral(const OpacityLaunch& L, cudaStream_t st0, int sms, void* scratch,
                            int64_t chunk_points, cudaStream_t aux, void* scratch1)
{
    if (L.npts <= 0 || L.n_energies <= 0)
        return cudaSuccess;
    const int ne     = L.n_energies;
    const int G      = pick_groups(ne < kEChunk ? ne : kEChunk, 2 * L.n1, 32);
    const bool pb    = L.use_pair || L.use_brem;
    const bool inel  = L.use_inel != 0;
    // With an auxiliary stream and scratch, consecutive chunks alternate
    // between the caller's stream and aux: the redo passes of one chunk (few
    // flagged records, a mostly idle grid) run beside the main passes of the
    // other.  The caller's stream waits for aux at the end.
    const bool two    = aux != nullptr && scratch1 != nullptr && L.npts > chunk_points;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    if (two)
    {
        cudaError_t e;
        if ((e = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaEventRecord(ev[0], st0)) != cudaSuccess ||
            (e = cudaStreamWaitEvent(aux, ev[0], 0)) != cudaSuccess)
        {
            if (ev[0])
                cudaEventDestroy(ev[0]);
            if (ev[1])
                cudaEventDestroy(ev[1]);
            return e;
        }
    }
    cudaError_t err = cudaSuccess;
    int64_t k       = 0;
    for (int64_t p0 = 0; p0 < L.npts && err == cudaSuccess; p0 += chunk_points, ++k)
    {
        const bool odd        = two && (k & 1);
        const cudaStream_t st = odd ? aux : st0;
        SpecPoint* pts        = (SpecPoint*)(odd ? scratch1 : scratch);
        uint64_t* fl_pb       = (uint64_t*)(pts + chunk_points);
        uint64_t* fl_nes      = fl_pb + chunk_points;
        EnergyRec* rec        = (EnergyRec*)(fl_nes + chunk_points);
        const int64_t np  = (L.npts - p0) < chunk_points ? (L.npts - p0) : chunk_points;
        phase_mark(kPhSpectral, 0, st);
        spec_prelude_kernel<<<(int)((np + 31) / 32), kPreTasks * 32, 0, st>>>(L, p0, np, pts);
        phase_mark(kPhSpectral, 1, st);
        if ((err = cudaGetLastError()) != cudaSuccess)
            break;
        if (!L.mixed)
        {
            if (pb && (err = launch_pb64(L, p0, np, pts, rec, nullptr, st)))
                break;
            if (inel && (err = launch_nes64(L, p0, np, pts, rec, nullptr, st)))
                break;
            err = launch_assemble<kSpecFp64>(L, p0, np, pts, rec, fl_pb, fl_nes, st, sms);
            continue;
        }
        if (pb && (err = launch_pb_mixed(L, p0, np, pts, rec, G, st, sms)))
            break;
        if (inel && (err = launch_nes_mixed(L, p0, np, pts, rec, st, sms)))
            break;
        if ((err = launch_assemble<kSpecMixed>(L, p0, np, pts, rec, fl_pb, fl_nes, st, sms)))
            break;
        for (int round = 0; round < 2 && err == cudaSuccess; ++round)
        {
            if (pb && (err = launch_pb64(L, p0, np, pts, rec, fl_pb, st)))
                break;
            if (inel && (err = launch_nes64(L, p0, np, pts, rec, fl_nes, st)))
                break;
            err = round == 0
                      ? launch_assemble<kSpecRedo>(L, p0, np, pts, rec, fl_pb, fl_nes, st, sms)
                      : launch_assemble<kSpecFinal>(L, p0, np, pts, rec, fl_pb, fl_nes, st, sms);
        }
    }
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
