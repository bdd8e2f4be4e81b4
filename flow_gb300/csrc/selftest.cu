// selftest.cu -- gb300_check_fp64_helpers and gb300_check_kernel_math: checks
// the integer-pipe and seeded arithmetic of the kernels (fused_math.cuh,
// exact_math.cuh, precision.cuh) against the IEEE operations on this GPU, over
// hashed inputs.
#include <cstring>

#include "../../include/flow_gb300.h"
#include "exact_math.cuh"
#include "fused_math.cuh"
#include "precision.cuh"

namespace flow {
namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

__device__ __forceinline__ bool same_value(double a, double b) {
  return (a != a && b != b) || dbits(a) == dbits(b);
}

// A normal double with a random mantissa, random sign and an exponent in
// [-60, 60].
__device__ __forceinline__ double normal_from(unsigned long long h) {
  const long long ex = 1023 - 60 + (long long)((h >> 52) % 121);
  return dfrom((long long)(h & 0x800fffffffffffffull) | (ex << 52));
}

__device__ __forceinline__ long long ulp_gap(double a, double b) {
  const long long d = dbits(a) - dbits(b);
  return d < 0 ? -d : d;
}

// counts[0] d_half != x*0.5, [1] d_twice != x*2 (all bit patterns, NaN = NaN),
// [2] d_is_pow2 wrong, [3] d_div != IEEE n/d, [4] d_rcp and a corrected quotient
// != IEEE n/d, [5] d_mul_pow2(x, 2^k) != x*2^k (all bit patterns of x, k in
// [-1022, 1023]); [6] the power-of-two quotients d_pow2_rcp, d_pow2_half_ratio,
// d_pow2_rcp_sq != 1/p, x/(2p), 1/(p*p) (exponents over the whole range); ulp[0],
// ulp[1] the largest gaps of [3], [4]; seed_err the largest |d_rcp_seed(d) d - 1|
// as FP64 bits.
__global__ void k_check(long long n, unsigned long long seed, unsigned long long* counts,
                        unsigned long long* ulp, unsigned long long* seed_err) {
  unsigned long long c[7] = {0, 0, 0, 0, 0, 0, 0}, u0 = 0, u1 = 0, se = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long h = mix64(seed ^ mix64((unsigned long long)i));
    // Bias three eighths of the patterns to the exponent-field ends (zeros,
    // subnormals, the smallest normals, the largest finite values, inf, NaN).
    unsigned long long b = h;
    const unsigned sel = (unsigned)(mix64(h) & 7u);
    if (sel == 0) b &= 0x801fffffffffffffull;                       // exponent 0 or 1
    if (sel == 1) b |= 0x7fe0000000000000ull;                       // exponent 0x7fe / 0x7ff
    if (sel == 2) b &= 0x8000000000000001ull;                       // zeros, tiny subnormal
    const double x = dfrom((long long)b);
    if (!same_value(d_half(x), __dmul_rn(x, 0.5))) ++c[0];
    if (!same_value(d_twice(x), __dmul_rn(x, 2.0))) ++c[1];
    int e2 = 0;
    const double m = frexp(x, &e2);
    const bool p2 = x > 0.0 && x <= 1.7976931348623157e308 && m == 0.5 && e2 >= -1021;
    if (d_is_pow2(x) != p2) ++c[2];
    // A power of two: mostly moderate exponents, an eighth over the whole range.
    const unsigned long long hp = mix64(h + 3);
    const long long kp = (hp & 7u) ? (long long)((hp >> 3) % 121) - 60
                                   : (long long)((hp >> 3) % 2046) - 1022;
    const double pw = dfrom((kp + 1023) << 52);
    if (!same_value(d_mul_pow2(x, pw), __dmul_rn(x, pw))) ++c[5];
    const unsigned long long hq = mix64(h + 4);
    const long long kq = (hq & 7u) ? (long long)((hq >> 3) % 121) - 60
                                   : (long long)((hq >> 3) % 2046) - 1022;
    const double pq = dfrom((kq + 1023) << 52);
    if (!same_value(d_pow2_rcp(pw), __ddiv_rn(1.0, pw))) ++c[6];
    if (!same_value(d_pow2_half_ratio(pq, pw), __ddiv_rn(pq, __dmul_rn(2.0, pw)))) ++c[6];
    if (!same_value(d_pow2_rcp_sq(pw), __ddiv_rn(1.0, __dmul_rn(pw, pw)))) ++c[6];
    const double nn = normal_from(mix64(h + 1)), dd = normal_from(mix64(h + 2));
    const double q = __ddiv_rn(nn, dd);
    const double qa = d_div(nn, dd);
    const double r = d_rcp(dd);
    const double qb = fma(r, fma(-dd, nn * r, nn), nn * r);
    if (dbits(qa) != dbits(q)) {
      ++c[3];
      const unsigned long long g = (unsigned long long)ulp_gap(qa, q);
      u0 = g > u0 ? g : u0;
    }
    if (dbits(qb) != dbits(q)) {
      ++c[4];
      const unsigned long long g = (unsigned long long)ulp_gap(qb, q);
      u1 = g > u1 ? g : u1;
    }
    const double err = fabs(fma(d_rcp_seed(dd), dd, -1.0));
    const unsigned long long eb = (unsigned long long)dbits(err);
    se = eb > se ? eb : se;
  }
  for (int k = 0; k < 7; ++k) {
    if (c[k]) atomicAdd(&counts[k], c[k]);
  }
  atomicMax(&ulp[0], u0);
  atomicMax(&ulp[1], u1);
  atomicMax(seed_err, se);
}

// A double of hash h, three eighths of them with an exponent at an end of the
// range (zeros, subnormals, the smallest normals, the largest values, inf, NaN).
__device__ __forceinline__ double end_biased(unsigned long long h) {
  unsigned long long b = h;
  const unsigned sel = (unsigned)(mix64(h) & 7u);
  if (sel == 0) b &= 0x801fffffffffffffull;
  if (sel == 1) b |= 0x7fe0000000000000ull;
  if (sel == 2) b &= 0x8000000000000001ull;
  return dfrom((long long)b);
}
__device__ __forceinline__ bool finite(double x) {
  return (dbits(x) & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
}

// The exact sum of eight doubles as hi + lo (two-sums; the parts below lo are
// below 2^-100 of the largest).
__device__ __forceinline__ void sum8_pair(const double (&v)[8], double& hi, double& lo) {
  hi = 0.0;
  lo = 0.0;
  for (int q = 0; q < 8; ++q) {
    const double s = __dadd_rn(hi, v[q]);
    const double bb = __dadd_rn(s, -hi);
    const double e = __dadd_rn(__dadd_rn(hi, -__dadd_rn(s, -bb)), __dadd_rn(v[q], -bb));
    hi = s;
    lo = __dadd_rn(lo, e);
  }
}

// Whether d_sum8 of eight values of one of four kinds is off: by more than the
// bits it drops (less than one unit of 2^-59 of the largest exponent a value)
// and its rounding, or of another class where a value is not finite.
__device__ __noinline__ bool sum8_wrong(unsigned long long h) {
  double v[8];
  const unsigned kind = (unsigned)(mix64(h + 40) & 3u);
  int emax = 0;
  bool fin = true;
  for (int q = 0; q < 8; ++q) {
    const unsigned long long hq = mix64(h + 50 + q);
    double x = normal_from(hq);
    if (kind == 0) x = dfrom((dbits(x) & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);
    if (kind == 2 && q >= 4) x = -dfrom(dbits(v[q - 4]) ^ (long long)(hq & 7u));
    if (kind == 3) x = end_biased(hq);
    v[q] = x;
    const int ex = (dhi(x) >> 20) & 0x7ff;
    emax = ex > emax ? ex : emax;
    fin = fin && finite(x);
  }
  const double got = d_sum8(v);
  const double plain = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  if (!fin) return (got != got) != (plain != plain) || (plain == plain && got != plain);
  if (emax < 64 || emax > 0x7f8) return !same_value(got, plain);  // (the additions)
  double hi, lo;
  sum8_pair(v, hi, lo);
  const double err = fabs(__dadd_rn(__dadd_rn(got, -hi), -lo));
  return !(err <= ldexp(1.0, emax - 1023 - 56) + fabs(got) * 1.1102230246251565e-16);
}

// counts[0] ex::div != IEEE n/d, [1] ex::slope != the products' minmod (zeros of
// either sign alike), [2] f32_diff != the FP64 difference, [3] f64_to_f32 or
// f32_to_f64 != the conversion (inside FP32's normal range), [4] d_sum8
// (sum8_wrong), [5] d_rcp != IEEE 1/x; gap the largest of [5] in units of the
// last place; seed_err the largest |d_rcp_seed(x) x - 1|, as FP64 bits, over
// every normal x whose reciprocal is normal.
__global__ void k_check_kernel_math(long long n, unsigned long long seed,
                                    unsigned long long* counts, unsigned long long* gap,
                                    unsigned long long* seed_err) {
  unsigned long long c[6] = {0, 0, 0, 0, 0, 0}, g = 0, se = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long h = mix64(seed ^ mix64((unsigned long long)i));
    // Half the quotients of neighbouring exponents, half of any.
    const double x = end_biased(h);
    double y = end_biased(mix64(h + 1));
    if (h & 16u) y = dfrom((dbits(y) & 0x800fffffffffffffLL) | (dbits(x) & 0x7ff0000000000000LL));
    if (!same_value(ex::div(x, y), __ddiv_rn(x, y))) ++c[0];
    // Differences alike in size, or of any.
    double b = end_biased(mix64(h + 2)), d = end_biased(mix64(h + 3));
    if (h & 32u) {
      const long long sx = dbits(x) & (long long)0xfff0000000000000ULL;
      b = dfrom((dbits(b) & 0x000fffffffffffffLL) | sx);
      d = dfrom((dbits(d) & 0x000fffffffffffffLL) | sx);
    }
    const double k = (h & 64u) ? fabs(normal_from(mix64(h + 4))) : fabs(end_biased(mix64(h + 4)));
    const double s0 = ex::slope(x, b, d, k), s1 = ex::slope_ieee(x, b, d, k);
    if (!same_value(s0, s1) && !(d_is_zero(s0) && d_is_zero(s1))) ++c[1];
    // Finite FP32 pairs: alike, a power of two apart, or of any size.
    unsigned fa = (unsigned)mix64(h + 5), fb = (unsigned)mix64(h + 6);
    if (h & 128u) fb = (fb & 0x807fffffu) | (fa & 0x7f800000u);
    if (h & 256u) fb = fa ^ ((fb & 31u) < 24u ? 1u << (fb & 31u) : 0u);
    if ((fa & 0x7f800000u) != 0x7f800000u && (fb & 0x7f800000u) != 0x7f800000u) {
      const float a = __uint_as_float(fa), e = __uint_as_float(fb);
      if (!same_value(f32_diff(a, e), __dadd_rn(f32_to_f64(a), -f32_to_f64(e)))) ++c[2];
      const double want = (fa & 0x7f800000u) ? (double)a : (a < 0.0f ? -0.0 : 0.0);
      if (f32_to_f64(a) != want) ++c[3];
    }
    {
      // An exponent in [-126, 127], one in eight with the ties' low bits.
      const long long ex = 1023 - 126 + (long long)((h >> 40) % 254);
      double w = dfrom((dbits(x) & (long long)0x800fffffffffffffULL) | (ex << 52));
      if ((h & 0x700u) == 0u) w = dfrom((dbits(w) & ~0x1fffffffLL) | 0x10000000LL);
      if (__float_as_uint(f64_to_f32(w)) != __float_as_uint(__double2float_rn(w))) ++c[3];
    }
    if (sum8_wrong(h)) ++c[4];
    const long long rex = 1 + (long long)((mix64(h + 7) >> 8) % 2043);  // 1 .. 2043
    const double r = dfrom((dbits(y) & (long long)0x800fffffffffffffULL) | (rex << 52));
    const double q = d_rcp(r), qi = __ddiv_rn(1.0, r);
    if (dbits(q) != dbits(qi)) {
      ++c[5];
      const unsigned long long gq = (unsigned long long)ulp_gap(q, qi);
      g = gq > g ? gq : g;
    }
    const unsigned long long eb =
        (unsigned long long)dbits(fabs(__fma_rn(d_rcp_seed(r), r, -1.0)));
    se = eb > se ? eb : se;
  }
  for (int k = 0; k < 6; ++k) {
    if (c[k]) atomicAdd(&counts[k], c[k]);
  }
  atomicMax(gap, g);
  atomicMax(seed_err, se);
}

}  // namespace
}  // namespace flow

extern "C" int gb300_check_kernel_math(long long n, unsigned long long seed, long long* counts,
                                       long long* max_rcp_ulp, double* max_seed_rel_err) {
  if (n <= 0 || !counts || !max_rcp_ulp || !max_seed_rel_err) return GB300_ERR_ARG;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 8 * sizeof(unsigned long long)) != cudaSuccess) return GB300_ERR_CUDA;
  cudaMemset(d, 0, 8 * sizeof(unsigned long long));
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  flow::k_check_kernel_math<<<sms * 8, 256>>>(n, seed, d, d + 6, d + 7);
  unsigned long long h[8];
  cudaError_t err = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) return GB300_ERR_CUDA;
  for (int k = 0; k < 6; ++k) counts[k] = (long long)h[k];
  *max_rcp_ulp = (long long)h[6];
  memcpy(max_seed_rel_err, &h[7], sizeof(double));
  return GB300_OK;
}

extern "C" int gb300_check_fp64_helpers(long long n, unsigned long long seed,
                                        long long* counts, long long* max_ulp,
                                        double* max_seed_rel_err) {
  if (n <= 0 || !counts || !max_ulp || !max_seed_rel_err) return GB300_ERR_ARG;
  unsigned long long* d = nullptr;
  if (cudaMalloc(&d, 10 * sizeof(unsigned long long)) != cudaSuccess) return GB300_ERR_CUDA;
  cudaMemset(d, 0, 10 * sizeof(unsigned long long));
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  flow::k_check<<<sms * 8, 256>>>(n, seed, d, d + 7, d + 9);
  unsigned long long h[10];
  cudaError_t err = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err != cudaSuccess) return GB300_ERR_CUDA;
  for (int k = 0; k < 7; ++k) counts[k] = (long long)h[k];
  max_ulp[0] = (long long)h[7];
  max_ulp[1] = (long long)h[8];
  double e;
  memcpy(&e, &h[9], sizeof(e));
  *max_seed_rel_err = e;
  return GB300_OK;
}
