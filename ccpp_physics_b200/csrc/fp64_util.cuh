// fp64_util.cuh -- FP64 helpers of the column kernels (lw_gas.cuh, lw_rt64.cuh,
// sw_column.cu): quotients without the IEEE slow path, table indices that
// equal the reference's, the split of the atmosphere, sums over lanes.
#pragma once
#include <cuda_runtime.h>

namespace fp64 {

// Quotients and roots from the hardware estimate (2^-20) and Newton's
// iteration, for operands that are normal numbers far from the ends of the
// range: no range check and no slow path, about two thirds of the instructions
// of the compiled IEEE operations.  recip_newton is 1/x to about 2^-52;
// div_markstein and sqrt_markstein add Markstein's residual step (IBM J. Res.
// Dev. 34, 1990), which rounds correctly but for a reciprocal whose own last
// bit was misrounded.
__device__ __forceinline__ double recip_newton(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
__device__ __forceinline__ double div_markstein(double a, double b) {
  const double y = recip_newton(b), q = a * y;
  return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ double sqrt_markstein(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(0.5 * y, fma(-x * y, y, 1.0), y);
  y = fma(0.5 * y, fma(-x * y, y, 1.0), y);
  const double r = x * y;
  return fma(fma(-r, r, x), 0.5 * y, r);
}
// int(z / (bpade + z) * 10000 + 0.5) (RSM:3601-3602, RLM:3602-3614), the index
// of the 10,001-entry transmittance tables, for 0 < z < 2^1022: beyond, the
// estimate is flushed to 0, so inputs without a bound of their own pass through
// finite_od first.  The quotient comes from one Newton step (error below
// 1e-8 in index units) and is rounded by adding 1.5 2^52; only a value within
// 1e-6 of a tie takes the IEEE division, so the entry is the reference's in every
// case.  NaN and infinity take it too, and the clamp, since the conversion of
// NaN is INT_MIN: index 0.
__device__ __forceinline__ int pade_index(double z) {
  constexpr double kBpade = 1.0 / 0.278, kRound = 6755399441055744.0;
  const double d = kBpade + z;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  y = fma(y, fma(-d, y, 1.0), y);
  const double q = z * y, t = fma(q, 10000.0, kRound);
  int i = __double2loint(t);
  const double f = fma(q, 10000.0, kRound - t);
  if (!(fabs(f) < 0.5 - 1.0e-6)) i = max(0, min(10000, (int)(z / d * 10000 + 0.5)));
  return i;
}

// A finite optical depth from 2^1000 on held there (opaque as well), so that
// neither it nor its slant path is out of the helpers' range; infinity and NaN
// stay.  By the high word.  (Range tests in pade_index, at all four lookups of a
// shortwave layer, cost the scheme 0.8 %, a branch around the layer's first
// quotients 0.7 %.)
__device__ __forceinline__ bool huge_od(double z) { return (unsigned)(__double2hiint(z) - 0x7e700000) < 0x01800000u; }
__device__ __forceinline__ double finite_od(double z) {
  return __hiloint2double(huge_od(z) ? 0x7e700000 : __double2hiint(z), __double2loint(z));
}

// ln p > 4.56 (the lower atmosphere, RLM:2344, RSM:2305): p against e^4.56 =
// 95.58347984, by the logarithm itself where rounding could decide.
__device__ __forceinline__ bool lower_atm(double p) {
  return (p > 95.5834 && p < 95.5836) ? log(p) > 4.56 : p > 95.5835;
}

// read-once inputs: no L1 line, which stays with exp_tbl
__device__ __forceinline__ double2 ld_once2(const double* p) {
  double2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

// Sums of N values (a power of two) over the L lanes (16 or 32) of a group:
// each step exchanges half of the values with the partner lane, so N values
// take N - 1 + log2(L / N) exchanges instead of N log2(L).  Lane j of the group
// ends with the sum of value sum_index<N, L>(j).
template <int N, int L>
__device__ __forceinline__ double lane_sums(double (&v)[N], int lane, unsigned mask) {
  int o = L / 2;
#pragma unroll
  for (int n = N / 2; n >= 1; n >>= 1, o >>= 1) {
    const bool hi = (lane & o) != 0;
#pragma unroll
    for (int q = 0; q < n; ++q) {
      const double keep = hi ? v[q + n] : v[q], send = hi ? v[q] : v[q + n];
      v[q] = keep + __shfl_xor_sync(mask, send, o);
    }
  }
  double r = v[0];
#pragma unroll
  for (; o >= 1; o >>= 1) r += __shfl_xor_sync(mask, r, o);
  return r;
}
// the value whose sum lane j of the group holds, -1 where another lane has it too
template <int N, int L>
__device__ __forceinline__ int sum_index(int lane) {
  int idx = 0, o = L / 2;
#pragma unroll
  for (int n = N / 2; n >= 1; n >>= 1, o >>= 1)
    if (lane & o) idx += n;
  return (lane & (2 * o - 1)) ? -1 : idx;
}

}  // namespace fp64
