// fused_math.cuh -- FP64 helpers of the fused timestep, shaped for GB300.
//
// On GB300 the FP64 pipe issues ~1.7 instructions per clock per SM, about
// 1/64 of the FP32 rate, while integer ALUs run at FP32-like rates.  DSETP
// comparisons occupy the FP64 pipe too.  So every comparison, sign test,
// absolute value, minimum and minmod selection here works on the IEEE bit
// pattern with integer instructions, and reciprocals / reciprocal square roots
// start from the MUFU approximation and finish with FMA Newton steps instead
// of the full IEEE division and square-root sequences.
//
// Semantics match the IEEE operations they replace for every finite input
// (including signed zeros); NaN inputs are not given IEEE ordering.
#pragma once

#include <cstdint>

namespace flow {

// Bit casts written as inline PTX moves, which the compiler cannot see
// through: with the plain intrinsics it folds integer tests such as
// "bits << 1 == 0" or "bits & ~sign" back into FP64 compares (DSETP) and
// absolute values, which occupy the FP64 pipe again.
__device__ __forceinline__ long long dbits(double x) {
  long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}
__device__ __forceinline__ double dfrom(long long b) {
  double x;
  asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
  return x;
}
__device__ __forceinline__ int dhi(double x) { return (int)(dbits(x) >> 32); }
__device__ __forceinline__ int dlo(double x) { return (int)dbits(x); }
__device__ __forceinline__ double dfrom2(int hi, int lo) {
  double x;
  asm("mov.b64 %0, {%1, %2};" : "=d"(x) : "r"(lo), "r"(hi));
  return x;
}
// -x with an integer instruction.
__device__ __forceinline__ double d_neg(double x) {
  return dfrom2(dhi(x) ^ (int)0x80000000, dlo(x));
}

__device__ __forceinline__ bool d_is_zero(double x) { return (dbits(x) << 1) == 0; }
// x > 0.0
__device__ __forceinline__ bool d_gt0(double x) { return dbits(x) > 0; }
// x < 0.0 (negative zero is not negative)
__device__ __forceinline__ bool d_lt0(double x) {
  const long long b = dbits(x);
  return b < 0 && (b << 1) != 0;
}
// x >= 0.0 (true for -0.0)
__device__ __forceinline__ bool d_ge0(double x) { return !d_lt0(x); }
__device__ __forceinline__ double d_abs(double x) {
  return dfrom(dbits(x) & 0x7fffffffffffffffLL);
}
// min(0.0, x) with the ordinary-minimum rule (first argument when smaller):
// 0.0 when x > 0, else x itself.
__device__ __forceinline__ double d_min0(double x) { return d_gt0(x) ? 0.0 : x; }
// Minimum of two non-negative values (bit patterns order like the values).
__device__ __forceinline__ double d_min_pos(double a, double b) {
  return (dbits(a) < dbits(b)) ? a : b;
}
// Slope limiter: the smaller-magnitude argument when both are non-zero with
// the same sign (the second on a tie), else +0.0.
__device__ __forceinline__ double d_minmod(double a, double b) {
  const long long ia = dbits(a), ib = dbits(b);
  const bool same = ((ia ^ ib) >= 0) && ((ia << 1) != 0) && ((ib << 1) != 0);
  const unsigned long long ma = (unsigned long long)ia & 0x7fffffffffffffffULL;
  const unsigned long long mb = (unsigned long long)ib & 0x7fffffffffffffffULL;
  return same ? ((ma < mb) ? a : b) : 0.0;
}

// x * 0.5 and x * 2 on the integer pipes, with the IEEE result for every
// input (zeros, subnormals, overflow to infinity, infinities and NaNs kept).
// For a normal x away from the range ends only the exponent field of the
// high word changes; at the low end the magnitude bits are linear in the
// value (exponent fields 0 and 1), so halving is a rounded shift.
__device__ __forceinline__ double d_half(double x) {
  const int hi = dhi(x);
  const unsigned ex = (unsigned)hi & 0x7ff00000u;
  if (ex - 0x00200000u < 0x7ff00000u - 0x00200000u) {
    return dfrom2(hi - 0x00100000, dlo(x));
  }
  const long long b = dbits(x);
  const long long mag = b & 0x7fffffffffffffffLL;
  if (mag >= 0x7ff0000000000000LL) return x;
  const long long h = (mag >> 1) + (mag & (mag >> 1) & 1);  // round half to even
  return dfrom((b ^ mag) | h);
}
__device__ __forceinline__ double d_twice(double x) {
  const int hi = dhi(x);
  const unsigned ex = (unsigned)hi & 0x7ff00000u;
  if (ex - 0x00100000u < 0x7fe00000u - 0x00100000u) {
    return dfrom2(hi + 0x00100000, dlo(x));
  }
  const long long b = dbits(x);
  const long long mag = b & 0x7fffffffffffffffLL;
  const long long sign = b ^ mag;
  if (ex == 0u) return dfrom(sign | (mag << 1));
  if (ex == 0x7fe00000u) return dfrom(sign | 0x7ff0000000000000LL);
  return x;
}
// x * p for p a positive normal power of two (an exact reciprocal of a
// power-of-two mesh spacing): an add to the exponent field when x and the
// result are normal, x itself for a zero; the rare rest (subnormal input or
// result, overflow, infinity, NaN) takes the FP64 multiply in a called
// function, so the common path issues no FP64 instruction.
static __device__ __noinline__ double d_mul_slow(double x, double p) { return __dmul_rn(x, p); }
__device__ __forceinline__ double d_mul_pow2(double x, double p) {
  const int hx = dhi(x);
  const int k = ((dhi(p) >> 20) & 0x7ff) - 1023;
  const int ex = (hx >> 20) & 0x7ff;
  if ((unsigned)(ex - 1) < 2046u && (unsigned)(ex + k - 1) < 2046u) {
    return dfrom2((int)((unsigned)hx + ((unsigned)k << 20)), dlo(x));
  }
  if ((dbits(x) << 1) == 0) return x;
  return d_mul_slow(x, p);
}
// True for a positive normal power of two (an exactly invertible spacing).
__device__ __forceinline__ bool d_is_pow2(double x) {
  const long long b = dbits(x);
  const unsigned ex = (unsigned)(b >> 52);  // sign bit lands above the field
  return (b & 0x000fffffffffffffLL) == 0 && ex - 1u < 0x7feu;
}
// r * e is exact and r * e / r gives e back: r a positive normal power of
// two, e a zero or a normal number whose product with r is normal (tests on
// the bit patterns, no FP64 instruction).
__device__ __forceinline__ bool d_pow2_product_exact(double r, double e) {
  const long long eb = dbits(e);
  const int ee = (int)((eb >> 52) & 0x7ff);
  const int ex = ee + (int)((dbits(r) >> 52) & 0x7ff) - 1023;
  return d_is_pow2(r) & (((eb << 1) == 0) | ((ee != 0) & (ee != 0x7ff) & (ex >= 1) & (ex <= 2046)));
}

// Quotients of powers of two, for the spacing factors of power-of-two
// meshes: 1/y, x/(2y) and 1/(y*y) with x, y positive normal powers of two.
// The quotient is a power of two itself, so when it is a normal number it
// is formed exactly from the exponent fields on the integer pipes (the IEEE
// quotient is that same number); otherwise the IEEE expression is evaluated
// in a called function.
static __device__ __noinline__ double d_pow2_quot_slow(double x, double y, int form) {
  if (form == 1) return x / (2.0 * y);
  if (form == 2) return 1.0 / (y * y);
  return 1.0 / y;
}
__device__ __forceinline__ int d_exp_field(double x) { return (dhi(x) >> 20) & 0x7ff; }
// 1/y
__device__ __forceinline__ double d_pow2_rcp(double y) {
  const int f = 2046 - d_exp_field(y);
  if ((unsigned)(f - 1) < 2046u) return dfrom2(f << 20, 0);
  return d_pow2_quot_slow(1.0, y, 0);
}
// x / (2 y)  (2 y must not overflow, as it is formed first)
__device__ __forceinline__ double d_pow2_half_ratio(double x, double y) {
  const int ey = d_exp_field(y);
  const int f = d_exp_field(x) - ey + 1022;
  if ((unsigned)(f - 1) < 2046u && ey < 2046) return dfrom2(f << 20, 0);
  return d_pow2_quot_slow(x, y, 1);
}
// 1 / (y * y)
__device__ __forceinline__ double d_pow2_rcp_sq(double y) {
  const int f = 3069 - 2 * d_exp_field(y);
  if ((unsigned)(f - 1) < 2046u) return dfrom2(f << 20, 0);
  return d_pow2_quot_slow(1.0, y, 2);
}

// 1/x to ~2^-43 for finite normal non-zero x, off the FP64 pipe: the mantissa
// as f + t 2^-23 in FP32 (f its first 24 bits, t the next 23), r0 the MUFU
// reciprocal of f, the Newton correction r0 (e + e^2) with e = 1 - (f + t
// 2^-23) r0 in FP32 FMAs, and r0 plus the correction (in units of 2^-43)
// assembled on the integer pipes.  About 30 FP32 and integer instructions in
// place of the two FP64 ones (128 clocks of a scheduler's FP64 issue) that
// bring the FP64 MUFU seed (2^-20) as far.
static __device__ __noinline__ double d_rcp_seed_slow(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return fma(r, fma(-x, r, 1.0), r);
}
__device__ __forceinline__ double d_rcp_seed(double x) {
  const int hi = dhi(x), lo = dlo(x);
  const int ex = (hi >> 20) & 0x7ff;
  // (The ends of the exponent range: the result would not be normal.)
  if ((unsigned)(ex - 1) >= 2043u) return d_rcp_seed_slow(x);
  const float f = __int_as_float(
      (int)(__funnelshift_l((unsigned)lo, (unsigned)hi, 3) & 0x7fffffu) | 0x3f800000);
  const float t = __int_as_float((int)(((unsigned)lo >> 6) & 0x7fffffu) | 0x3f800000) - 1.0f;
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(f));
  r0 = fminf(fmaxf(r0, 0.5f), 1.0f);  // (f lies in [1, 2); its last place aside, so does 1/r0)
  float e = fmaf(-f, r0, 1.0f);
  e = fmaf(-t, r0 * 1.1920928955078125e-7f, e);
  const float r1 = r0 * fmaf(e, e, e);  // |r1| < 2^-21
  constexpr float kMagic = 1.430511474609375e-6f;  // 1.5 2^-20: units of 2^-43
  const int k = __float_as_int(r1 + kMagic) - __float_as_int(kMagic);
  const unsigned b = (unsigned)__float_as_int(r0);
  // r0 widened, its exponent less x's, plus k 2^-43 (r0's last place is 2^-53).
  const long long m = ((long long)(int)((b >> 3) + (unsigned)((896 + 1023 - ex) << 20)) << 32) +
                      (long long)(unsigned)(b << 29) + ((long long)k << 10);
  return dfrom2((int)(m >> 32) ^ (hi & (int)0x80000000), (int)m);
}
// 1/x for finite normal non-zero x: MUFU seed, two Newton-Raphson steps (the
// mixed form's spacing factors, once per tile).
__device__ __forceinline__ double d_rcp_newton(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}
// 1/x for finite normal non-zero x: the seed and one Newton step.
__device__ __forceinline__ double d_rcp(double x) {
  const double r = d_rcp_seed(x);
  return fma(r, fma(-x, r, 1.0), r);
}
// n/d for finite normal non-zero d when 1/d itself is not needed: the quotient
// from the seed and one residual correction q + r (n - d q) (2^-43 -> ~2^-86):
// the correctly rounded quotient except in vanishingly rare near-ties, in 3
// FP64 instructions (5 with a Newton step on the MUFU seed).
__device__ __forceinline__ double d_div(double n, double d) {
  const double r = d_rcp_seed(d);
  const double q = n * r;
  return fma(r, fma(-d, q, n), q);
}
// 1/sqrt(x) for finite normal positive x: MUFU seed, two Newton steps on
// r <- r + r*(0.5 - 0.5*x*r*r).
__device__ __forceinline__ double d_rsqrt(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double h = d_half(x);
  double t = fma(-h * r, r, 0.5);
  r = fma(r, t, r);
  t = fma(-h * r, r, 0.5);
  return fma(r, t, r);
}

// Writes the value of interior point (ii, jj) of a w x h array into each of
// its ghost mirror images (pad layers per side): column images negated when
// flip_x, row images when flip_y, corner images by both.  This reproduces the
// reflective fill of every ghost point whose mirror source is (ii, jj).
__device__ __forceinline__ void mirror_store(double* a, int w, int h, int pad,
                                             int ii, int jj, double val,
                                             bool flip_x, bool flip_y) {
  int mc[2], mr[2];
  int nc = 0, nr = 0;
  if (jj < 2 * pad) mc[nc++] = 2 * pad - 1 - jj;
  if (jj >= w - 2 * pad) mc[nc++] = 2 * (w - pad) - 1 - jj;
  if (ii < 2 * pad) mr[nr++] = 2 * pad - 1 - ii;
  if (ii >= h - 2 * pad) mr[nr++] = 2 * (h - pad) - 1 - ii;
  if (nc == 0 && nr == 0) return;
  const double vx = flip_x ? -val : val;
  const double vy = flip_y ? -val : val;
  const double vxy = flip_x ? -vy : vy;
  for (int k = 0; k < nc; ++k) a[(size_t)ii * w + mc[k]] = vx;
  for (int r = 0; r < nr; ++r) {
    a[(size_t)mr[r] * w + jj] = vy;
    for (int k = 0; k < nc; ++k) a[(size_t)mr[r] * w + mc[k]] = vxy;
  }
}

// The sum of eight doubles on the integer pipes, rounded once: their
// mantissas, aligned to the largest exponent with 7 more bits, added as 64-bit
// integers (60 bits and 3 for the sum).  Bits of a value more than 59 places
// below the largest's leading one are dropped, well below the rounding of an
// FP64 addition at that size.  About 85 integer instructions (two clocks of a
// scheduler each) in place of eight additions of 64 clocks: the totals' two
// FP64 instructions a cell bound them (16.4 M cells: 58 us of FP64 issue, 39
// us of memory).  Infinities, NaNs and the ends of the exponent range take the
// additions (a call, so that the others do not issue them).
static __device__ __noinline__ double d_sum8_slow(double a, double b, double c, double d, double e,
                                                  double f, double g, double h) {
  return ((a + b) + (c + d)) + ((e + f) + (g + h));
}
__device__ __forceinline__ double d_sum8(const double (&v)[8]) {
  int emax = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int ex = (dhi(v[q]) >> 20) & 0x7ff;
    emax = ex > emax ? ex : emax;
  }
  if (emax > 0x7f8 || emax < 64) {
    return d_sum8_slow(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
  }
  long long sum = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long b = dbits(v[q]);
    const int ex = (int)((b >> 52) & 0x7ff);
    const int sh = emax - ex;
    // (A zero or subnormal, which has no leading one, lies below the alignment.)
    const unsigned long long m =
        (((unsigned long long)b & 0x000fffffffffffffULL) | 0x0010000000000000ULL) << 7;
    const long long a = sh < 60 ? (long long)(m >> sh) : 0;
    sum += b < 0 ? -a : a;
  }
  if (sum == 0) return 0.0;
  const bool neg = sum < 0;
  unsigned long long m = neg ? 0ull - (unsigned long long)sum : (unsigned long long)sum;
  const int lz = __clzll((long long)m);  // leading one at bit 63 - lz
  m <<= lz;
  // Round to nearest even at bit 11.
  const unsigned long long r = (m >> 11) + (((m & 0x7ffULL) + ((m >> 11) & 1ULL)) > 0x400ULL);
  // m at bit 59 has the exponent emax; r holds the leading one at bit 52 (or
  // carried to 53), which the sum adds to the exponent field below it.
  const long long e = (long long)(emax + (63 - lz) - 59 - 1);
  return dfrom((long long)((unsigned long long)(e << 52) + r) |
               (neg ? (long long)0x8000000000000000ULL : 0LL));
}

}  // namespace flow
