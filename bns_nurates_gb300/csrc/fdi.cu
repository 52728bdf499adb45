// Batched Fermi-Dirac integrals of the reference's family (functions.hpp:442-4375):
// F_j(x) = integral_0^inf t^j / (exp(t - x) + 1) dt without the 1 / Gamma(j + 1)
// normalisation, j = k2 / 2 for k2 = -9, -7, -5, -3, -1 (FDI_m92 .. FDI_m12,
// continued below j = -1 by dF_{j+1}/dx = (j + 1) F_j) and k2 = 0 .. 21
// (FDI_0, FDI_p12, FDI_p1, ..., FDI_p10, FDI_p212).
//
// Integer orders 0..5 run the fixed-point Taylor tables of bnsn_fx.cuh.  Every
// other order is a factor times one polynomial of degree 15 in the tables of
// bnsn_fdi_tab.h (made by fdi_tables.py from mpmath): the alternating series in
// e^x below x = -4, one of 70 intervals of [-4, 100), the Sommerfeld expansion
// above.  The tables agree with the reference's approximations to a few 1e-16
// (relative, away from the zeros of the negative orders).
//
// Non-finite arguments follow the reference: NaN gives NaN for the
// half-integer orders and 0 for the integer ones; -inf gives 0; +inf gives
// +inf for j > -1 and -0 or +0 (the sign of x^(j+1) / (j+1)) below.
//
// One thread per argument, grid-stride, the order's table (9 KB) in shared memory
// per CTA.  Arguments come in any order, so a warp usually meets all three regimes:
// they share the polynomial, and the factors (e^x, x^(j+1)) run on the integer
// pipes (bnsn_fx.cuh).  The interval and the position in it come from the argument in
// fixed point.  FP64-pipe bound, ~20 operations per argument against 16 bytes of traffic.
// A loop per regime instead (16 + 25 Clenshaw + 12 terms, exp, sqrt and two
// divisions) cost a mixed warp the sum of them: ~150.  4,000,037 arguments uniform in
// [-50, 150), order 1/2: 978 -> 164 us (265 with the interval in FP64).

#include <cuda_runtime.h>

#include "bnsn_fdi_tab.h"
#include "bnsn_fp64.cuh"
#include "bnsn_internal.h"

namespace bnsn {
namespace {

using namespace fp64;

// Table slot of a twice-order (kTwice[slot] == k2), -1 when not tabulated.
constexpr int slot_of(int k2)
{
    for (int s = 0; s < fdit::kNumOrders; ++s)
        if (fdit::kTwice[s] == k2)
            return s;
    return -1;
}

// One order's coefficients in shared memory, [term][row]: the lanes of a warp read the
// same term of different rows.
struct FdiShared
{
    double c[fdit::kDegree + 1][fdit::kRows];
};

// x^(h/2) for x >= 100 (or +inf) and |h| <= 23 outside the fixed-point range (x >
// 2^120 or a result that leaves the exponent range): an integer power by repeated
// squaring, times sqrt(x) for odd h, inverted for negative h.
__device__ __noinline__ double pow_half(double x, int h)
{
    const int a = h < 0 ? -h : h;
    int q       = a >> 1;
    double v = 1., b = x;
    while (q)
    {
        if (q & 1)
            v *= b;
        q >>= 1;
        if (q)
            b *= b;
    }
    if (a & 1)
        v *= sqrt(x);
    return h < 0 ? 1. / v : v;
}

// P = j + 1 in 2^-58 units, ij1 = 1 / (j + 1).
__device__ __forceinline__ double fdi_table(const FdiShared& S, int h, int64_t P, double ij1,
                                            bool integer, double x)
{
    using namespace fdit;
    static_assert(kXlo == -4. && kXmid == 40. && kXhi == 100. && kWidth == 11. / 16. &&
                      kWide == 10. && kNarrow == 64,
                  "fx::fd_interval");
    const uint64_t bits = fx::bits_of(x), mag = bits & 0x7fffffffffffffffull;
    const bool neg      = (int64_t)bits < 0;
    double v, f = 1.;
    int row;
    if (neg && mag > 0x4010000000000000ull) // x < -4, or NaN
    {
        f   = fx::exp(x);
        v   = -f;
        row = 0;
    }
    else if (!neg && mag >= 0x4059000000000000ull) // x >= 100, or NaN
    {
        row = kPieces + 1;
        if (mag < 0x44f0000000000000ull) // 2^80
        {
            const int64_t L = fx::log2_q56(x);
            v = fx::pow_q(L, -2 * (1ll << 58));
            f = fx::pow_q(L, P) * ij1;
        }
        else
        {
            v = 1. / (x * x);
            f = pow_half(x, h) * ij1;
        }
    }
    else
    {
        v = fx::fd_interval(x, &row);
        ++row;
    }
    double p = S.c[kDegree][row];
#pragma unroll
    for (int m = kDegree - 1; m >= 0; --m)
        p = fma(p, v, S.c[m][row]);
    // NaN: 0 for the integer orders, as the reference's regime tests give
    return mag > 0x7ff0000000000000ull ? (integer ? 0. : x) : f * p;
}

template <int K>
__global__ void fdi_int_kernel(const double* __restrict__ x, double* __restrict__ out, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = fdi<K>(x[i]);
}

__global__ void fdi_table_kernel(int slot, int h, int integer, const double* __restrict__ x,
                                 double* __restrict__ out, int64_t n)
{
    using namespace fdit;
    __shared__ FdiShared S;
    for (int k = threadIdx.x; k < kRows * (kDegree + 1); k += blockDim.x)
    {
        const int row = k / (kDegree + 1), m = k - row * (kDegree + 1);
        S.c[m][row] = kPoly[slot][row][m];
    }
    const int64_t P  = fx::pow_exponent(0.5 * h);
    const double ij1 = 2. / h;
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = fdi_table(S, h, P, ij1, integer != 0, x[i]);
}

} // namespace

// Twice-orders the family defines: -9, -7, -5, -3, -1 and 0 .. 21.
bool fdi_order_valid(int k2) { return (k2 >= 0 && k2 <= 21) || (k2 < 0 && k2 >= -9 && (k2 & 1)); }

cudaError_t launch_fdi(int k2, const double* x, double* out, int64_t n, cudaStream_t stream,
                       int num_sms)
{
    if (n <= 0)
        return cudaSuccess;
    constexpr int threads = 256;
    const int64_t need    = (n + threads - 1) / threads;
    const int64_t cap     = (int64_t)num_sms * 8;
    const int grid        = (int)(need < cap ? need : cap);
    const int slot        = slot_of(k2);
    if (slot < 0 && !(k2 >= 0 && k2 <= 10 && (k2 & 1) == 0))
        return cudaErrorInvalidValue;
    phase_mark(kPhAux, 0, stream);
    switch (k2)
    {
    case 0: fdi_int_kernel<0><<<grid, threads, 0, stream>>>(x, out, n); break;
    case 2: fdi_int_kernel<1><<<grid, threads, 0, stream>>>(x, out, n); break;
    case 4: fdi_int_kernel<2><<<grid, threads, 0, stream>>>(x, out, n); break;
    case 6: fdi_int_kernel<3><<<grid, threads, 0, stream>>>(x, out, n); break;
    case 8: fdi_int_kernel<4><<<grid, threads, 0, stream>>>(x, out, n); break;
    case 10: fdi_int_kernel<5><<<grid, threads, 0, stream>>>(x, out, n); break;
    default:
        fdi_table_kernel<<<grid, threads, 0, stream>>>(slot, k2 + 2, (k2 & 1) == 0, x, out, n);
    }
    phase_mark(kPhAux, 1, stream);
    return cudaGetLastError();
}

} // namespace bnsn
