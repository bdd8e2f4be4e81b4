// exact_math.cuh -- IEEE operations of the bit-exact stage kernels (stages.cu),
// off the FP64 pipe where it can be.  The FP64 pipe issues one warp instruction
// per 64 clocks and scheduler, and comparisons, selections and the sequence of
// an IEEE division (eight FP64 instructions and more) run on it too.  Every
// function here returns the bits of the C expression it stands for (a NaN is a
// NaN; a zero may differ in sign where stated).
#pragma once

#include "fused_math.cuh"

namespace flow {
namespace ex {

constexpr long long kInf = 0x7ff0000000000000LL;

// x > 0.0, x >= 0.0, x != 0.0 (false, false, true for a NaN)
__device__ __forceinline__ bool gt0(double x) {
  const long long b = dbits(x);
  return b > 0 && b <= kInf;
}
__device__ __forceinline__ bool ge0(double x) {
  const long long b = dbits(x);
  return (b >= 0 && b <= kInf) || (b << 1) == 0;
}
__device__ __forceinline__ bool nz(double x) { return !d_is_zero(x); }
// (0.0 < x) ? 0.0 : x
__device__ __forceinline__ double min0(double x) { return gt0(x) ? 0.0 : x; }
// Slope limiter: the argument of smaller magnitude when both are non-zero and
// of the same sign (the second on a tie), else +0.0 (also for a NaN).
__device__ __forceinline__ double minmod(double a, double b) {
  const long long ia = dbits(a), ib = dbits(b);
  const long long ma = ia & 0x7fffffffffffffffLL, mb = ib & 0x7fffffffffffffffLL;
  const bool ok = (ia ^ ib) >= 0 && ma != 0 && mb != 0 && ma <= kInf && mb <= kInf;
  return ok ? (ma < mb ? a : b) : 0.0;
}

// The limited slope minmod(minmod(0.5 k a, 2 k b), 2 k c) of three differences,
// k = 1/h, with the products formed as the reference does, (0.5 k) a.  Where
// halving and doubling are exact for a, b, c and k the scaling can follow the
// selection: (0.5 k) a and k (0.5 a) then round the same number, and rounding
// keeps the order of the magnitudes.  Near the ends of the exponent range
// (half of a subnormal difference rounds, twice a large one overflows) the
// products are formed one by one.
static __device__ __noinline__ double slope_ieee(double a, double b, double c, double k) {
  const double h = __dmul_rn(0.5, k), t = __dmul_rn(2.0, k);
  return minmod(minmod(__dmul_rn(h, a), __dmul_rn(t, b)), __dmul_rn(t, c));
}
// Exponent fields 4 .. 2043.
__device__ __forceinline__ bool mid_range(double x) {
  return (unsigned)(dhi(x) & 0x7fffffff) - 0x00400000u < 0x7f800000u;
}
__device__ __forceinline__ double slope(double a, double b, double c, double k) {
  const bool ok = mid_range(k) && (mid_range(a) || d_is_zero(a)) &&
                  (mid_range(b) || d_is_zero(b)) && (mid_range(c) || d_is_zero(c));
  if (!ok) return slope_ieee(a, b, c, k);
  return __dmul_rn(minmod(minmod(d_half(a), d_twice(b)), d_twice(c)), k);
}

// n / d.  The quotient from the 2^-43 seed with one residual correction, then
// its exact residual t = n - d q: q is the correctly rounded quotient when |t|
// is less than |d| times half a unit of q's last place (no quotient of two
// doubles lies halfway; a power of two, whose lower neighbour is nearer, does
// not take this test).  A few in 2^33 fail it, and they and operands near the
// ends of the exponent range take the IEEE division.  Four FP64 instructions
// where the IEEE sequence takes eight or more.
static __device__ __noinline__ double div_ieee(double n, double d) { return __ddiv_rn(n, d); }
__device__ __forceinline__ double div(double n, double d) {
  const int en = (dhi(n) >> 20) & 0x7ff, ed = (dhi(d) >> 20) & 0x7ff;
  if ((unsigned)(ed - 128) < 1792u) {
    if (d_is_zero(n)) return dfrom2((dhi(n) ^ dhi(d)) & (int)0x80000000, 0);
    if ((unsigned)(en - 128) < 1792u && (unsigned)(en - ed + 895) < 1792u) {
      const double r = d_rcp_seed(d);
      double q = __dmul_rn(n, r);
      q = __fma_rn(r, __fma_rn(-d, q, n), q);
      const long long qb = dbits(q);
      const long long t = dbits(__fma_rn(-d, q, n)) & 0x7fffffffffffffffLL;
      const long long eq = (qb >> 52) & 0x7ff;
      const long long bound = (dbits(d) & 0x7fffffffffffffffLL) + ((eq - 1076) << 52);
      if (t == 0 || (t < bound && (qb & 0x000fffffffffffffLL) != 0)) return q;
    }
  }
  return div_ieee(n, d);
}
// n / h and x * h for a mesh spacing h: exponent adds where p2 (h a power of
// two; ih is 1/h then).
__device__ __forceinline__ double div_h(double n, double h, double ih, bool p2) {
  return p2 ? d_mul_pow2(n, ih) : div(n, h);
}
__device__ __forceinline__ double mul_h(double x, double h, bool p2) {
  return p2 ? d_mul_pow2(x, h) : __dmul_rn(x, h);
}

}  // namespace ex
}  // namespace flow
