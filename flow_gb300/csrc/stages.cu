// stages.cu -- the per-function kernels of the GB300 flow kernel set.
//
// One kernel per loop of the reference timestep (omp3/flow.c) plus the device
// ghost fill, the CFL minimum and the conservation totals.  These back the
// individual entry points of omp3/flow.h:4-88 (equation_of_state,
// pressure_acceleration, ...), so that a host driver can call any stage on its
// own, and they form the "exact" timestep: this file is compiled without
// floating-point contraction (--fmad=false) and evaluates every expression in
// the reference's order, so each entry point reproduces the reference's IEEE
// results bit for bit.  The fused, faster timestep lives in fused.cu.
//
// Every kernel is a 2-D launch: x over columns (coalesced), y over rows.
#include <atomic>

#include "common.cuh"
#include "exact_math.cuh"
#include "precision.cuh"
#include "stages.h"

namespace flow {
namespace {

constexpr int kBX = 64;
constexpr int kBY = 4;

inline dim3 grid_for(int rows, int cols) {
  return dim3((unsigned)((cols + kBX - 1) / kBX),
              (unsigned)((rows + kBY - 1) / kBY));
}
// The stage kernels are launched with programmatic stream serialisation: a
// kernel's blocks start while its predecessor's last ones run, and wait here
// for it to complete before they touch memory (after any other predecessor the
// wait returns at once).  A step is some thirty launches, most of them of a few
// microseconds: 3.63 -> 3.35 ms for four steps at 1280x1024.  Every
// predecessor of a waiting kernel has itself waited, so the order is the
// stream's.
__device__ __forceinline__ void stage_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" :::);
}
template <typename... KArgs, typename... Args>
void launch_stage(void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}
#define FLOW_POINT(i0, i1, j0, j1)                                   \
  stage_begin();                                                     \
  const int jj = (j0) + (int)(blockIdx.x * blockDim.x + threadIdx.x); \
  const int ii = (i0) + (int)(blockIdx.y * blockDim.y + threadIdx.y); \
  if (ii >= (i1) || jj >= (j1)) return;

// A mesh spacing with its power-of-two test and, where it holds, its reciprocal
// (exact).  The kernels below evaluate the reference's expressions with the
// operations of exact_math.cuh: the same bits with about half of the FP64
// instructions (1280x1024, four steps with totals: 11485 us before, 4458 after).
struct Spacing {
  double h, ih;
  bool p2;
  __device__ __forceinline__ explicit Spacing(double v)
      : h(v), ih(0.0), p2(d_is_pow2(v) && d_exp_field(v) < 2000 && d_exp_field(v) > 40) {
    if (p2) ih = d_pow2_rcp(v);
  }
  __device__ __forceinline__ double div(double n) const { return ex::div_h(n, h, ih, p2); }
  __device__ __forceinline__ double mul(double x) const { return ex::mul_h(x, h, p2); }
  __device__ __forceinline__ double rcp() const { return p2 ? ih : ex::div(1.0, h); }
};

// Volume-weighted density on an x-face / y-face (omp3/flow.c:134-141).
__device__ __forceinline__ double rho_xface(int nx, const double* rho,
                                            const double* edgedx,
                                            const double* celldx,
                                            const double* celldy, int ii,
                                            int jj) {
  const Spacing cy(celldy[ii]), c1(celldx[jj]), c0(celldx[jj - 1]);
  return ex::div(cy.mul(c1.mul(rho[cidx(nx, ii, jj)])) +
                     cy.mul(c0.mul(rho[cidx(nx, ii, jj - 1)])),
                 cy.mul(d_twice(edgedx[jj])));
}
__device__ __forceinline__ double rho_yface(int nx, const double* rho,
                                            const double* edgedy,
                                            const double* celldx,
                                            const double* celldy, int ii,
                                            int jj) {
  const Spacing cx(celldx[jj]), c1(celldy[ii]), c0(celldy[ii - 1]);
  return ex::div(c1.mul(cx.mul(rho[cidx(nx, ii, jj)])) +
                     c0.mul(cx.mul(rho[cidx(nx, ii - 1, jj)])),
                 Spacing(edgedy[ii]).mul(d_twice(celldx[jj])));
}

// ---------------------------------------------------------------------------
// Lagrangian phase.

__global__ void k_eos(int nx, int ny, double* P, const double* rho,
                      const double* e) {
  FLOW_POINT(0, ny, 0, nx);
  const size_t c = cidx(nx, ii, jj);
  P[c] = (kGam - 1.0) * rho[c] * e[c];
}

// Pressure (viscous = 0) or viscous-stress (viscous = 1) acceleration of the
// face momenta followed by the velocity update (omp3/flow.c:121-152 and
// 212-240): the two loops differ only in the force and its spacing.
template <int kViscous>
__global__ void k_accelerate(int nx, int ny, int pad, double dt,
                             double* rho_u, double* rho_v, double* u, double* v,
                             const double* fx, const double* fy,
                             const double* rho, const double* edgedx,
                             const double* edgedy, const double* celldx,
                             const double* celldy) {
  FLOW_POINT(pad, (ny + 1) - pad, pad, (nx + 1) - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  const Spacing hx(kViscous ? celldx[jj] : edgedx[jj]);
  const Spacing hy(kViscous ? celldy[ii] : edgedy[ii]);
  const double mu = rho_u[f] - hx.div(dt * (fx[c] - fx[c - 1]));
  const double mv = rho_v[c] - hy.div(dt * (fy[c] - fy[c - nx]));
  rho_u[f] = mu;
  rho_v[c] = mv;
  const double rx = rho_xface(nx, rho, edgedx, celldx, celldy, ii, jj);
  const double ry = rho_yface(nx, rho, edgedy, celldx, celldy, ii, jj);
  u[f] = ex::nz(rx) ? ex::div(mu, rx) : 0.0;
  v[c] = ex::nz(ry) ? ex::div(mv, ry) : 0.0;
}

// Limited compressive velocity jumps (omp3/flow.c:177-198).
__device__ __forceinline__ void visc_jumps(double lo, double mid, double hi,
                                           double hi2, double* jump,
                                           double* curv) {
  const double j0 = ex::min0(mid - lo), j1 = ex::min0(hi - mid), j2 = ex::min0(hi2 - hi);
  *jump = j1;
  *curv = d_half(d_abs(j2 - j1) + d_abs(j1 - j0));
}

__global__ void k_viscous_stress(int nx, int ny, int pad, double* Qxx,
                                 double* Qyy, const double* u, const double* v,
                                 const double* rho) {
  FLOW_POINT(pad, ny - pad, pad, nx - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  double u_i, u_ii, v_i, v_ii;
  visc_jumps(u[f - 1], u[f], u[f + 1], u[f + 2], &u_i, &u_ii);
  visc_jumps(v[c - nx], v[c], v[c + nx], v[c + 2 * nx], &v_i, &v_ii);
  const double cr = -kCQ * rho[c];
  Qxx[c] = cr * u_i * u_ii;
  Qyy[c] = cr * v_i * v_ii;
}

__global__ void k_shock_heating(int nx, int ny, int pad, double dt_h,
                                double* e, const double* P, const double* u,
                                const double* v, const double* rho,
                                const double* Qxx, const double* Qyy,
                                const double* celldx, const double* celldy) {
  FLOW_POINT(pad, ny - pad, pad, nx - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  const double r = rho[c];
  const double p = P[c];
  const double dudx = Spacing(celldx[jj]).div(u[f + 1] - u[f]);
  const double dvdy = Spacing(celldy[ii]).div(v[c + nx] - v[c]);
  const double div_dt = (dudx + dvdy) * dt_h;
  const double e_q = e[c] - ex::div(dt_h * (Qxx[c] * dudx + Qyy[c] * dvdy), r);
  const double rho_c = ex::div(r, 1.0 + div_dt);
  const double e_c = e_q - ex::div(p * div_dt, r);
  const double work = ex::div(d_half(div_dt) * (p + (kGam - 1.0) * e_c * rho_c), r);
  e[c] = ex::nz(r) ? e_q - work : 0.0;
}

// ---------------------------------------------------------------------------
// Reductions: per-thread partials over a grid-stride range of interior cells,
// warp shuffles, one partial per block in reduce_array, and the last block to
// finish combines the partials (single pass, no second launch).

__device__ __forceinline__ double warp_min(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = dmin(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

constexpr int kRedThreads = 256;

// Leapfrog update of omp3/flow.c:103-105 from the global CFL minimum g.
__device__ __forceinline__ void apply_dt_rule(double g, double dt_h_in, int first_step,
                                              double* ra) {
  const double limited = dmin(g, FLOW_C_M * dt_h_in);
  const double dt = 0.5 * (kCT * limited + dt_h_in);
  ra[kRaDt] = dt;
  ra[kRaDtH] = first_step ? dt : kCT * limited;
}

// The timestep candidates of one cell (omp3/flow.c:80-90).
__device__ __forceinline__ double cfl_candidate(double e, double q, double rho, double h) {
  const double sound = sqrt(kGam * (kGam - 1.0) * e);
  return h / sqrt(sound * sound + 2.0 * q / rho);
}

// The smallest candidate of a block's cells, each thread's from its first cell
// t on in strides: m where it is smaller, else m.  A candidate costs about 45
// FP64 instructions (two square roots and two quotients), and nearly every one
// is larger than the smallest by far, so a first pass ranks the cells in FP32
// by S / h^2 = 1/dt^2 (S = c_s^2 + 2 Q / rho), and the second evaluates
//   - among the cells without viscous stress, only the largest energy: every
//     operation of the candidate rounds monotonically, so it is the smallest;
//   - of the others those within 1e-4 of the block's largest FP32 rank, whose
//     error is below 1e-5.
// Returns false, with nothing done, for a block with a cell the ranks do not
// hold for (negative, infinite or NaN energy or stress, a density that is not
// positive and normal, ranks outside FP32's middle range, or spacings that are
// not all one number): its cells are all evaluated.  (1280x1024: 224 us with
// every cell evaluated; the step 1110 us, 907 with the ranks and paired fills.)
__device__ __forceinline__ bool ranked_min(int w, long long n, int nx, int pad, const double* Qxx,
                                           const double* Qyy, const double* rho, const double* e,
                                           const double* celldx, const double* celldy, double* m) {
  __shared__ unsigned s_rank;
  __shared__ unsigned long long s_ex, s_ey;
  const double hx = celldx[pad], hy = celldy[pad];
  const float ix = 1.0f / f64_to_f32(hx), iy = 1.0f / f64_to_f32(hy);
  const float kx = ix * ix, ky = iy * iy;
  const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long step = (long long)gridDim.x * blockDim.x;
  if (threadIdx.x == 0) {
    s_rank = 0u;
    s_ex = s_ey = 0ull;
  }
  // The larger rank of the cell, negative where the ranks do not hold; each
  // axis's own in rx, ry.  The narrowing turns a stress below 2^-126 into zero,
  // which takes up to 2^-126 ir from the cell's S: less than 1e-5 of an S above
  // 1.2e-33 ir.  (A stress of 1e-39 sets the timestep where the density is
  // 1e-25 and the energy 1e-15.)  S and the squares of the reciprocal spacings
  // are normal FP32 numbers too, so that no step but the narrowing loses bits.
  const bool mid = kx > 1e-30f && kx < 1e30f && ky > 1e-30f && ky < 1e30f;
  auto rank = [&](double ec, double qx, double qy, double r, float& rx, float& ry) {
    const long long be = dbits(ec), bx = dbits(qx), by = dbits(qy), br = dbits(r);
    const float ef = f64_to_f32(ec), rf = f64_to_f32(r), ir = 2.0f / rf;
    const float sx = fmaf(f64_to_f32(qx), ir, 0.56f * ef);
    const float sy = fmaf(f64_to_f32(qy), ir, 0.56f * ef);
    rx = sx * kx;
    ry = sy * ky;
    const bool ok = be >= 0 && be < ex::kInf && (bx >= 0 || (bx << 1) == 0) && bx < ex::kInf &&
                    (by >= 0 || (by << 1) == 0) && by < ex::kInf &&
                    (unsigned long long)br - 0x0010000000000000ULL < 0x7fe0000000000000ULL;
    const float k = fmaxf(rx, ry);
    return ok && mid && k > 1e-30f && k < 1e30f && rf > 1e-30f && rf < 1e30f &&
                   fminf(sx, sy) > fmaxf(1e-30f, 2e-33f * ir)
               ? k
               : -1.0f;
  };
  bool ok = true;
  float best = 0.0f;
  for (long long t = t0; t < n; t += step) {
    const int ii = pad + (int)(t / w), jj = pad + (int)(t % w);
    const size_t c = cidx(nx, ii, jj);
    float rx, ry;
    const float k = rank(e[c], Qxx[c], Qyy[c], rho[c], rx, ry);
    ok = ok && k >= 0.0f && dbits(celldx[jj]) == dbits(hx) && dbits(celldy[ii]) == dbits(hy);
    best = fmaxf(best, k);
  }
  if (!__syncthreads_and(ok)) return false;
  atomicMax(&s_rank, __float_as_uint(best));  // (non-negative: ordered as integers)
  __syncthreads();
  const float bound = __uint_as_float(s_rank) * 0.9999f;
  unsigned long long ex_x = 0ull, ex_y = 0ull;  // bits of the largest energies, plus one
  for (long long t = t0; t < n; t += step) {
    const int ii = pad + (int)(t / w), jj = pad + (int)(t % w);
    const size_t c = cidx(nx, ii, jj);
    const double ec = e[c], qx = Qxx[c], qy = Qyy[c], r = rho[c];
    float rx, ry;
    rank(ec, qx, qy, r, rx, ry);
    const unsigned long long be = (unsigned long long)dbits(ec) + 1ull;
    if (d_is_zero(qx)) {
      ex_x = be > ex_x ? be : ex_x;
    } else if (rx >= bound) {
      *m = dmin(*m, cfl_candidate(ec, qx, r, hx));
    }
    if (d_is_zero(qy)) {
      ex_y = be > ex_y ? be : ex_y;
    } else if (ry >= bound) {
      *m = dmin(*m, cfl_candidate(ec, qy, r, hy));
    }
  }
  if (ex_x) atomicMax(&s_ex, ex_x);
  if (ex_y) atomicMax(&s_ey, ex_y);
  __syncthreads();
  if (threadIdx.x == 0) {
    // (Without stress 2 Q / rho is a zero.)
    if (s_ex) *m = dmin(*m, cfl_candidate(dfrom((long long)(s_ex - 1)), 0.0, 1.0, hx));
    if (s_ey) *m = dmin(*m, cfl_candidate(dfrom((long long)(s_ey - 1)), 0.0, 1.0, hy));
  }
  return true;
}

// local_only: a rank of a decomposed mesh keeps its minimum in ra[kRaMinBits]
// (the caller reduces it over the ranks and applies the rule, k_dt_rule).
__global__ void __launch_bounds__(kRedThreads)
    k_min_timestep(int nx, int ny, int pad, double max_dt, double dt_h_in,
                   int first_step, const double* Qxx, const double* Qyy,
                   const double* rho, const double* e, const double* celldx,
                   const double* celldy, double* ra, int local_only) {
  const int w = nx - 2 * pad;
  const long long n = (long long)w * (ny - 2 * pad);
  double m = max_dt;
  if (!ranked_min(w, n, nx, pad, Qxx, Qyy, rho, e, celldx, celldy, &m)) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
      const int ii = pad + (int)(t / w);
      const int jj = pad + (int)(t % w);
      const size_t c = cidx(nx, ii, jj);
      const double cfl_x = cfl_candidate(e[c], Qxx[c], rho[c], celldx[jj]);
      const double cfl_y = cfl_candidate(e[c], Qyy[c], rho[c], celldy[ii]);
      m = dmin(m, dmin(cfl_x, cfl_y));
    }
  }
  __shared__ double s_part[kRedThreads / 32];
  __shared__ bool s_last;
  m = warp_min(m);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    double x = (threadIdx.x < kRedThreads / 32) ? s_part[threadIdx.x] : max_dt;
    x = warp_min(x);
    if (threadIdx.x == 0) {
      ra[kRaPartial + blockIdx.x] = x;
      __threadfence();
      unsigned long long* ticket = reinterpret_cast<unsigned long long*>(ra + kRaTicket);
      s_last = (atomicAdd(ticket, 1ull) == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double x = max_dt;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    x = dmin(x, __ldcg(ra + kRaPartial + b));
  }
  x = warp_min(x);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    double g = s_part[0];
    for (int k = 1; k < kRedThreads / 32; ++k) g = dmin(g, s_part[k]);
    if (local_only) {
      ra[kRaMinBits] = g;
    } else {
      apply_dt_rule(g, dt_h_in, first_step, ra);
    }
    *reinterpret_cast<unsigned long long*>(ra + kRaTicket) = 0ull;
  }
}

__global__ void k_dt_rule(double g, double dt_h_in, int first_step, double* ra) {
  if (threadIdx.x == 0) apply_dt_rule(g, dt_h_in, first_step, ra);
}

// Partial sums of one thread: two (mass, energy) pairs.
struct ConsSums {
  double m0, e0, m1, e1;
};

// The FP64 work of the conservation sums sits in calls, so that a warp that
// skips it skips its instructions (a predicated FP64 instruction still takes
// its issue slots on the FP64 pipe).  plain: bit q set where group q is summed.
__device__ __noinline__ ConsSums cons_add_groups(ConsSums s, unsigned plain, double d0,
                                                 double d1, double d2, double d3, double f0,
                                                 double f1, double f2, double f3) {
  if (plain & 1u) {
    s.m0 += d0;
    s.e0 = fma(d0, f0, s.e0);
  }
  if (plain & 2u) {
    s.m1 += d1;
    s.e1 = fma(d1, f1, s.e1);
  }
  if (plain & 4u) {
    s.m0 += d2;
    s.e0 = fma(d2, f2, s.e0);
  }
  if (plain & 8u) {
    s.m1 += d3;
    s.e1 = fma(d3, f3, s.e1);
  }
  return s;
}
// A run of n groups of 32 cells holding one (rho, e) pair: n*rho and
// n*(rho*e) per lane.
__device__ __noinline__ ConsSums cons_add_run(ConsSums s, int n, unsigned long long r_bits,
                                              unsigned long long e_bits) {
  const double dn = (double)n, r = __longlong_as_double(r_bits);
  s.m1 += dn * r;
  s.e1 += dn * (r * __longlong_as_double(e_bits));
  return s;
}

// The interior is cut into chunks of 4 x 256 columns of one row (each warp
// 4 groups of 32 consecutive cells) and the chunks are dealt to the blocks in
// turn: a block loads its next chunk before it sums the current one (16 loads
// of independent columns in flight per thread), into two pairs of sums, rho*e
// contracted into one FMA -- two FP64 instructions per cell, the FP64 pipe's
// share of this reduction on GB300.  The grid is one wave of resident blocks.
// Columns past the last whole chunk of a row (rows whose interior is not a
// multiple of 1024 wide) are summed after the chunks, by 256-column groups
// and a ragged end.  A group whose 32 cells hold one (rho, e) pair (bit for
// bit; the fluid at rest around a blast) is counted instead: the warp keeps
// the pair of its current run of such groups and their number, and adds
// n*rho and n*(rho*e) per lane when the run ends -- integer work in place of
// 64 FP64 instructions per group, and the same sum to rounding.
constexpr int kConsChunk = 4 * kRedThreads;

__global__ void __launch_bounds__(kRedThreads)
    k_conservation(int nx, int ny, int pad, const double* __restrict__ rho,
                   const double* __restrict__ e, double* ra) {
  ConsSums acc{0.0, 0.0, 0.0, 0.0};
  unsigned long long run_r = 0ull, run_e = 0ull;  // warp-uniform
  int run_n = 0;
  // Group q of 32 cells of a warp: counted into the run (returns 0), or to be
  // summed (returns bit q).
  auto group = [&](double d, double f, int q) -> unsigned {
    const unsigned long long db = __double_as_longlong(d), fb = __double_as_longlong(f);
    const unsigned long long d0 = __shfl_sync(0xffffffffu, db, 0);
    const unsigned long long f0 = __shfl_sync(0xffffffffu, fb, 0);
    if (!__all_sync(0xffffffffu, db == d0 && fb == f0)) return 1u << q;
    if (d0 != run_r || f0 != run_e) {
      if (run_n > 0) acc = cons_add_run(acc, run_n, run_r, run_e);
      run_r = d0;
      run_e = f0;
      run_n = 0;
    }
    ++run_n;
    return 0u;
  };
  const int w = nx - 2 * pad, rows = ny - 2 * pad;
  const int t = threadIdx.x;
  const int per_row = w / kConsChunk;
  const long long chunks = (long long)rows * per_row;
  double d[4], f[4];
  auto load = [&](long long c, double* dd, double* ff) {
    const int r = (int)(c / per_row);
    const size_t base = (size_t)(pad + r) * nx + pad + (size_t)(c - (long long)r * per_row) * kConsChunk + t;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      dd[q] = rho[base + q * kRedThreads];
      ff[q] = e[base + q * kRedThreads];
    }
  };
  long long c = blockIdx.x;
  if (c < chunks) load(c, d, f);
  while (c < chunks) {
    const long long cn = c + gridDim.x;
    double dn[4], fn[4];
    if (cn < chunks) load(cn, dn, fn);
    unsigned plain = 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) plain |= group(d[q], f[q], q);
    if (plain) acc = cons_add_groups(acc, plain, d[0], d[1], d[2], d[3], f[0], f[1], f[2], f[3]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      d[q] = dn[q];
      f[q] = fn[q];
    }
    c = cn;
  }
  if (per_row * kConsChunk < w) {
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
      const double* rr = rho + (size_t)(pad + r) * nx + pad;
      const double* er = e + (size_t)(pad + r) * nx + pad;
      int j0 = per_row * kConsChunk;
      for (; j0 + kRedThreads <= w; j0 += kRedThreads) {
        const double dd = rr[j0 + t], ff = er[j0 + t];
        if (group(dd, ff, 0)) acc = cons_add_groups(acc, 1u, dd, 0.0, 0.0, 0.0, ff, 0.0, 0.0, 0.0);
      }
      if (j0 + t < w) {
        acc.m0 += rr[j0 + t];
        acc.e0 = fma(rr[j0 + t], er[j0 + t], acc.e0);
      }
    }
  }
  if (run_n > 0) acc = cons_add_run(acc, run_n, run_r, run_e);
  double ms = acc.m0 + acc.m1, es = acc.e0 + acc.e1;
  __shared__ double s_m[kRedThreads / 32], s_e[kRedThreads / 32];
  __shared__ bool s_last;
  ms = warp_sum(ms);
  es = warp_sum(es);
  if ((threadIdx.x & 31) == 0) {
    s_m[threadIdx.x >> 5] = ms;
    s_e[threadIdx.x >> 5] = es;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int k = 0; k < kRedThreads / 32; ++k) {
      a += s_m[k];
      b += s_e[k];
    }
    ra[kRaPartial + 2 * blockIdx.x] = a;
    ra[kRaPartial + 2 * blockIdx.x + 1] = b;
    __threadfence();
    unsigned long long* ticket = reinterpret_cast<unsigned long long*>(ra + kRaTicket);
    s_last = (atomicAdd(ticket, 1ull) == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double a = 0.0, b = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    a += __ldcg(ra + kRaPartial + 2 * k);
    b += __ldcg(ra + kRaPartial + 2 * k + 1);
  }
  a = warp_sum(a);
  b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) {
    s_m[threadIdx.x >> 5] = a;
    s_e[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tb = 0.0;
    for (int k = 0; k < kRedThreads / 32; ++k) {
      ta += s_m[k];
      tb += s_e[k];
    }
    ra[kRaMass] = ta;
    ra[kRaEnergy] = tb;
    *reinterpret_cast<unsigned long long*>(ra + kRaTicket) = 0ull;
  }
}

// ---------------------------------------------------------------------------
// Mass and energy advection (omp3/flow.c:326-554).  kDirY selects the sweep:
// x fluxes live on x-faces (stride nx+1), y fluxes on y-faces (stride nx).

template <int kDirY>
__global__ void k_mass_energy_flux(int nx, int ny, int pad, double dt,
                                   double dt_h, const double* rho,
                                   const double* e, const double* vel,
                                   double* F, double* eF, const double* celldx,
                                   const double* edgedx, const double* celldy,
                                   const double* edgedy) {
  FLOW_POINT(pad, kDirY ? (ny + 1) - pad : ny - pad, pad,
             kDirY ? nx - pad : (nx + 1) - pad);
  const size_t c = cidx(nx, ii, jj);
  const size_t fv = kDirY ? c : fidx(nx, ii, jj);  // index of the face
  const ptrdiff_t sv = kDirY ? nx : 1;             // velocity stride
  const ptrdiff_t sc = kDirY ? nx : 1;             // cell stride
  const double invd = Spacing(kDirY ? edgedy[ii] : edgedx[jj]).rcp();
  const double wm = vel[fv - sv], w0 = vel[fv], wp = vel[fv + sv];
  const double slope = ex::slope(wp - wm, w0 - wm, wp - w0, invd);
  const double w_tc = w0 - d_half(w0) * dt * slope;

  const double r_m2 = rho[c - 2 * sc], r_m1 = rho[c - sc], r_0 = rho[c],
               r_p1 = rho[c + sc];
  double limiter = 0.0;
  const double rho_jump = (r_0 - r_m1);
  if (ex::nz(rho_jump)) {  // also true for NaN, as `if (x)` in C
    // The y sweep takes the smoothness side from v itself (omp3/flow.c:477).
    const double side = kDirY ? w0 : w_tc;
    const bool up = ex::ge0(side);
    const double smooth = ex::div((up ? r_m1 : r_p1) - (up ? r_m2 : r_0), rho_jump);
    limiter = ex::div(smooth + d_abs(smooth), 1.0 + d_abs(smooth));
  }
  const bool ge = ex::ge0(w_tc), pos = ex::gt0(w_tc);
  const double rho_up = ge ? r_m1 : r_0;
  const Spacing h0(kDirY ? celldy[ii] : celldx[jj]);
  const double hm = kDirY ? celldy[ii - 1] : celldx[jj - 1];
  const double wdt = w_tc * dt_h;
  const double flux =
      (w_tc * rho_up +
       d_half(d_abs(w_tc)) * (1.0 - d_abs(h0.div(wdt))) * limiter * rho_jump);
  F[fv] = flux;

  const double e_m2 = e[c - 2 * sc], e_m1 = e[c - sc], e_0 = e[c],
               e_p1 = e[c + sc];
  // The side the wind comes from: the reference evaluates both.
  const double base = pos ? e_m1 : e_0, far = pos ? e_m2 : e_m1, near = pos ? e_0 : e_p1;
  const double m = ex::slope(near - far, base - far, near - base, invd);
  const double hs = d_half(m) * (pos ? hm - wdt : h0.h + wdt);
  const double e_face = pos ? base + hs : base - hs;
  const double area = kDirY ? edgedx[jj] : edgedy[ii];
  eF[fv] = area * e_face * flux;
}

template <int kDirY>
__global__ void k_mass_energy_update(int nx, int ny, int pad, int first,
                                     double dt_h, double* rho,
                                     const double* rho_old, double* e,
                                     const double* F, const double* eF,
                                     const double* celldx, const double* edgedx,
                                     const double* celldy,
                                     const double* edgedy) {
  FLOW_POINT(pad, ny - pad, pad, nx - pad);
  const size_t c = cidx(nx, ii, jj);
  const size_t f0 = kDirY ? c : fidx(nx, ii, jj);
  const size_t f1 = kDirY ? c + nx : f0 + 1;
  // The x sweep weights both faces by edgedy of rows ii+1 and ii, the y sweep
  // by edgedx of columns jj+1 and jj (omp3/flow.c:417-418, 533-534).
  const double a1 = kDirY ? edgedx[jj + 1] : edgedy[ii + 1];
  const double a0 = kDirY ? edgedx[jj] : edgedy[ii];
  const Spacing vol(celldx[jj] * celldy[ii]);
  const double r_new = rho[c] - vol.div(dt_h * (a1 * F[f1] - a0 * F[f0]));
  rho[c] = r_new;
  const double r_old = rho_old[c];
  const double rho_e = r_old * e[c] - vol.div(dt_h * (eF[f1] - eF[f0]));
  const double denom = first ? r_old : r_new;
  e[c] = ex::nz(denom) ? ex::div(rho_e, denom) : 0.0;
}

// ---------------------------------------------------------------------------
// Momentum advection (omp3/flow.c:557-970).

__device__ __forceinline__ double mc_upwind(double wind, double m2, double m1,
                                            double p0, double p1, double invd,
                                            double d_left, double d_right,
                                            double dt_h, double lm, double rp) {
  // The side the wind comes from (the reference evaluates both).
  const bool pos = ex::gt0(wind);
  const double base = pos ? lm : rp, far = pos ? m2 : m1, mid = pos ? m1 : p0,
               near = pos ? p0 : p1;
  const double m = ex::slope(near - far, mid - far, near - mid, invd);
  const double wdt = wind * dt_h;
  const double hs = d_half(m) * (pos ? d_left - wdt : d_right + wdt);
  return pos ? base + hs : base - hs;
}

// uF_x: cell-centred x flux of rho u (omp3/flow.c:778-823).
__global__ void k_uF_x(int nx, int ny, int pad, double dt_h, const double* u,
                       double* uF_x, const double* F_x, const double* edgedx,
                       const double* edgedy, const double* celldx) {
  FLOW_POINT(pad, ny - pad, pad, nx - pad);
  const size_t f = fidx(nx, ii, jj);
  const double invdx = Spacing(edgedx[jj]).rcp();
  const double u_cell = d_half(u[f] + u[f + 1]);
  const double mass = d_half(edgedy[ii]) * (F_x[f] + F_x[f + 1]);
  const double u_up = mc_upwind(u_cell, u[f - 1], u[f], u[f + 1], u[f + 2],
                                invdx, celldx[jj - 1], celldx[jj], dt_h, u[f],
                                u[f + 1]);
  uF_x[cidx(nx, ii, jj)] = mass * u_up;
}

// uF_y: corner y flux of rho u (omp3/flow.c:826-874).
__global__ void k_uF_y(int nx, int ny, int pad, double dt_h, const double* u,
                       const double* v, double* uF_y, const double* F_y,
                       const double* edgedx, const double* edgedy,
                       const double* celldy) {
  FLOW_POINT(pad, (ny + 1) - pad, pad, (nx + 1) - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  const ptrdiff_t r = nx + 1;
  const double invdy = Spacing(edgedy[ii]).rcp();
  const double v_corner = d_half(v[c - 1] + v[c]);
  const double mass = d_half(edgedx[jj]) * (F_y[c] + F_y[c - 1]);
  const double u_up = mc_upwind(v_corner, u[f - 2 * r], u[f - r], u[f],
                                u[f + r], invdy, celldy[ii - 1], celldy[ii],
                                dt_h, u[f - r], u[f]);
  uF_y[f] = mass * u_up;
}

// vF_x: corner x flux of rho v (omp3/flow.c:877-925).
__global__ void k_vF_x(int nx, int ny, int pad, double dt_h, const double* u,
                       const double* v, double* vF_x, const double* F_x,
                       const double* edgedx, const double* celldy,
                       const double* celldx) {
  FLOW_POINT(pad, (ny + 1) - pad, pad, (nx + 1) - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  const ptrdiff_t r = nx + 1;
  const double invdx = Spacing(edgedx[jj]).rcp();
  const double mass = d_half(celldy[ii]) * (F_x[f] + F_x[f - r]);
  const double u_corner = d_half(u[f] + u[f - r]);
  const double v_up = mc_upwind(u_corner, v[c - 2], v[c - 1], v[c], v[c + 1],
                                invdx, celldx[jj - 1], celldx[jj], dt_h,
                                v[c - 1], v[c]);
  vF_x[f] = mass * v_up;
}

// vF_y: cell-centred y flux of rho v (omp3/flow.c:928-970).
__global__ void k_vF_y(int nx, int ny, int pad, double dt_h, const double* v,
                       double* vF_y, const double* F_y, const double* edgedy,
                       const double* celldx, const double* celldy) {
  FLOW_POINT(pad, ny - pad, pad, nx - pad);
  const size_t c = cidx(nx, ii, jj);
  const double invdy = Spacing(edgedy[ii]).rcp();
  const double mass = d_half(celldx[jj]) * (F_y[c] + F_y[c + nx]);
  const double v_cell = d_half(v[c] + v[c + nx]);
  const double v_up = mc_upwind(v_cell, v[c - nx], v[c], v[c + nx],
                                v[c + 2 * nx], invdy, celldy[ii - 1],
                                celldy[ii], dt_h, v[c], v[c + nx]);
  vF_y[c] = mass * v_up;
}

// Momentum updates (omp3/flow.c:577-668, 683-771).  kWhich: 0 rho_u by uF_x,
// 1 rho_u by uF_y, 2 rho_v by vF_x, 3 rho_v by vF_y.
template <int kWhich>
__global__ void k_momentum_update(int nx, int ny, int pad, double dt_h,
                                  int with_vel, double* mom, double* vel,
                                  const double* flux, const double* rho,
                                  const double* edgedx, const double* edgedy,
                                  const double* celldx, const double* celldy) {
  constexpr bool kU = (kWhich < 2);
  FLOW_POINT(pad, kU ? ny - pad : (ny + 1) - pad, pad,
             kU ? (nx + 1) - pad : nx - pad);
  const size_t f = fidx(nx, ii, jj);
  const size_t c = cidx(nx, ii, jj);
  const size_t at = kU ? f : c;
  double df, area;
  if (kWhich == 0) {
    df = flux[c] - flux[c - 1];
    area = edgedx[jj] * celldy[ii];
  } else if (kWhich == 1) {
    df = flux[f + (nx + 1)] - flux[f];
    area = celldx[jj] * edgedy[ii];
  } else if (kWhich == 2) {
    df = flux[f + 1] - flux[f];
    area = edgedx[jj] * celldy[ii];
  } else {
    df = flux[c] - flux[c - nx];
    area = celldx[jj] * edgedy[ii];
  }
  const double m = mom[at] - Spacing(area).div(dt_h * df);
  mom[at] = m;
  if (with_vel) {
    const double r = kU ? rho_xface(nx, rho, edgedx, celldx, celldy, ii, jj)
                        : rho_yface(nx, rho, edgedy, celldx, celldy, ii, jj);
    vel[at] = ex::nz(r) ? ex::div(m, r) : 0.0;
  }
}

// ---------------------------------------------------------------------------
// Reflective ghost fill of one w x h array (the arch handle_boundary_2d of a
// single rank).  Every ghost point takes the value of its mirror image in the
// interior, negated once per mirrored axis that is inverted; this equals
// filling the x walls over the interior rows and then copying whole rows for
// the y walls.  Needs at least `pad` interior points per axis.
__device__ __forceinline__ void boundary_point(long long t, int w, int h, int pad, double* arr,
                                               int flip_x, int flip_y) {
  const long long n_rows = 2LL * pad * w;
  const long long n_cols = 2LL * pad * (h - 2 * pad);
  if (t >= n_rows + n_cols) return;
  int ii, jj;
  if (t < n_rows) {
    const int r = (int)(t / w);
    jj = (int)(t % w);
    ii = (r < pad) ? r : h - 2 * pad + r;
  } else {
    const long long s = t - n_rows;
    const int r = (int)(s / (2 * pad));
    const int k = (int)(s % (2 * pad));
    ii = pad + r;
    jj = (k < pad) ? k : w - 2 * pad + k;
  }
  int si = ii, sj = jj;
  bool neg = false;
  if (jj < pad) { sj = 2 * pad - 1 - jj; neg ^= (flip_x != 0); }
  else if (jj >= w - pad) { sj = 2 * (w - pad) - 1 - jj; neg ^= (flip_x != 0); }
  if (ii < pad) { si = 2 * pad - 1 - ii; neg ^= (flip_y != 0); }
  else if (ii >= h - pad) { si = 2 * (h - pad) - 1 - ii; neg ^= (flip_y != 0); }
  const double val = arr[(size_t)si * w + sj];
  arr[(size_t)ii * w + jj] = neg ? -val : val;
}

__global__ void k_boundary(int w, int h, int pad, double* arr, int flip_x, int flip_y) {
  stage_begin();
  boundary_point(blockIdx.x * (long long)blockDim.x + threadIdx.x, w, h, pad, arr, flip_x, flip_y);
}
// Two arrays in one launch (blockIdx.y): a fill of a few hundred KB takes 4 to 5
// us, most of it the launch.
__global__ void k_boundary2(int w0, int h0, double* a0, int flip_x0, int flip_y0, int w1, int h1,
                            double* a1, int flip_x1, int flip_y1, int pad) {
  stage_begin();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (blockIdx.y == 0) boundary_point(t, w0, h0, pad, a0, flip_x0, flip_y0);
  else boundary_point(t, w1, h1, pad, a1, flip_x1, flip_y1);
}

// The x-wall part of the reflective fill (ghost columns of the interior rows)
// on the sides whose bit is set in sides (1 west, 2 east), and the y-wall part
// (whole ghost rows, x ghosts included) on sides 4 south (low rows), 8 north.
// With all four bits, the x part followed by the y part fills exactly what
// k_boundary fills.
__global__ void k_reflect_x(int w, int h, int pad, double* arr, int flip_x, int sides) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 2LL * pad * (h - 2 * pad)) return;
  const int r = (int)(t / (2 * pad));
  const int k = (int)(t % (2 * pad));
  const int ii = pad + r;
  if (k < pad) {
    if (!(sides & 1)) return;
    const int jj = k;
    const double val = arr[(size_t)ii * w + (2 * pad - 1 - jj)];
    arr[(size_t)ii * w + jj] = flip_x ? -val : val;
  } else {
    if (!(sides & 2)) return;
    const int jj = w - 2 * pad + k;
    const double val = arr[(size_t)ii * w + (2 * (w - pad) - 1 - jj)];
    arr[(size_t)ii * w + jj] = flip_x ? -val : val;
  }
}
__global__ void k_reflect_y(int w, int h, int pad, double* arr, int flip_y, int sides) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= 2LL * pad * w) return;
  const int r = (int)(t / w);
  const int jj = (int)(t % w);
  if (r < pad) {
    if (!(sides & 4)) return;
    const double val = arr[(size_t)(2 * pad - 1 - r) * w + jj];
    arr[(size_t)r * w + jj] = flip_y ? -val : val;
  } else {
    if (!(sides & 8)) return;
    const int ii = h - 2 * pad + r;
    const double val = arr[(size_t)(2 * (h - pad) - 1 - ii) * w + jj];
    arr[(size_t)ii * w + jj] = flip_y ? -val : val;
  }
}

__global__ void k_copy(size_t n, double* dst, const double* src) {
  stage_begin();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    dst[i] = src[i];
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host launchers.

#define FLOW_LAUNCH2D(kern, rows, cols, ...)                         \
  do {                                                               \
    if ((rows) > 0 && (cols) > 0) {                                  \
      launch_stage(kern, grid_for((rows), (cols)), dim3(kBX, kBY), s, __VA_ARGS__); \
    }                                                                \
  } while (0)

void launch_eos(cudaStream_t s, int nx, int ny, double* P, const double* rho,
                const double* e) {
  FLOW_LAUNCH2D(k_eos, ny, nx, nx, ny, P, rho, e);
}

void launch_accelerate(cudaStream_t s, bool viscous, int nx, int ny, int pad,
                       double dt, double* rho_u, double* rho_v, double* u,
                       double* v, const double* fx, const double* fy,
                       const double* rho, const MeshView& m) {
  const int rows = (ny + 1) - 2 * pad, cols = (nx + 1) - 2 * pad;
  if (viscous) {
    FLOW_LAUNCH2D(k_accelerate<1>, rows, cols, nx, ny, pad, dt, rho_u, rho_v, u,
                  v, fx, fy, rho, m.edgedx, m.edgedy, m.celldx, m.celldy);
  } else {
    FLOW_LAUNCH2D(k_accelerate<0>, rows, cols, nx, ny, pad, dt, rho_u, rho_v, u,
                  v, fx, fy, rho, m.edgedx, m.edgedy, m.celldx, m.celldy);
  }
}

void launch_viscous_stress(cudaStream_t s, int nx, int ny, int pad, double* Qxx,
                           double* Qyy, const double* u, const double* v,
                           const double* rho) {
  FLOW_LAUNCH2D(k_viscous_stress, ny - 2 * pad, nx - 2 * pad, nx, ny, pad, Qxx,
                Qyy, u, v, rho);
}

void launch_shock_heating(cudaStream_t s, int nx, int ny, int pad, double dt_h,
                          double* e, const double* P, const double* u,
                          const double* v, const double* rho, const double* Qxx,
                          const double* Qyy, const MeshView& m) {
  FLOW_LAUNCH2D(k_shock_heating, ny - 2 * pad, nx - 2 * pad, nx, ny, pad, dt_h,
                e, P, u, v, rho, Qxx, Qyy, m.celldx, m.celldy);
}

int reduce_blocks(int nx, int ny, int pad, int partials_per_block) {
  const long long cells = (long long)(nx - 2 * pad) * (ny - 2 * pad);
  const long long cap = ((long long)nx * ny - kRaPartial) / partials_per_block;
  long long b = (cells + kRedThreads - 1) / kRedThreads;
  if (b > kMaxReduceBlocks) b = kMaxReduceBlocks;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// One wave of resident conservation blocks on the current device (the SM
// count and the kernel's occupancy, looked up once per device), no more than
// the chunks and rows to deal out nor the partial slots of reduce_array.
int conservation_blocks(int nx, int ny, int pad) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> wave[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  int b = (dev >= 0 && dev < kMaxDevices) ? wave[dev].load(std::memory_order_relaxed) : 0;
  if (b == 0) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_conservation, kRedThreads, 0);
    b = sms * per_sm > 0 ? sms * per_sm : kMaxReduceBlocks;
    if (dev >= 0 && dev < kMaxDevices) wave[dev].store(b, std::memory_order_relaxed);
  }
  const int w = nx - 2 * pad, rows = ny - 2 * pad;
  long long work = (long long)rows * (w / kConsChunk);  // whole chunks
  if (work < rows) work = rows;  // rows of ragged ends
  const long long cap = ((long long)nx * ny - kRaPartial) / 2;
  long long g = b;
  if (g > work) g = work;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

void launch_min_timestep(cudaStream_t s, int nx, int ny, int pad, double max_dt,
                         double dt_h, int first_step, const double* Qxx,
                         const double* Qyy, const double* rho, const double* e,
                         const MeshView& m, double* reduce_array, int local_only) {
  cudaMemsetAsync(reduce_array + kRaTicket, 0, sizeof(double), s);
  k_min_timestep<<<reduce_blocks(nx, ny, pad, 1), kRedThreads, 0, s>>>(
      nx, ny, pad, max_dt, dt_h, first_step, Qxx, Qyy, rho, e, m.celldx,
      m.celldy, reduce_array, local_only);
}

void launch_dt_rule(cudaStream_t s, double g, double dt_h, int first_step, double* ra) {
  k_dt_rule<<<1, 32, 0, s>>>(g, dt_h, first_step, ra);
}

void launch_reflect_x(cudaStream_t s, int w, int h, int pad, double* arr, int invert,
                      int sides) {
  const long long n = 2LL * pad * (h - 2 * pad);
  if (n <= 0 || !(sides & 3)) return;
  k_reflect_x<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, h, pad, arr, invert == kInvertX,
                                                         sides);
}

void launch_reflect_y(cudaStream_t s, int w, int h, int pad, double* arr, int invert,
                      int sides) {
  const long long n = 2LL * pad * w;
  if (n <= 0 || !(sides & 12)) return;
  k_reflect_y<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, h, pad, arr, invert == kInvertY,
                                                         sides);
}

void launch_conservation(cudaStream_t s, int nx, int ny, int pad,
                         const double* rho, const double* e,
                         double* reduce_array) {
  cudaMemsetAsync(reduce_array + kRaTicket, 0, sizeof(double), s);
  k_conservation<<<conservation_blocks(nx, ny, pad), kRedThreads, 0, s>>>(
      nx, ny, pad, rho, e, reduce_array);
  count_launches(1);
}

void launch_mass_energy_flux(cudaStream_t s, bool dir_y, int nx, int ny,
                             int pad, double dt, double dt_h, const double* rho,
                             const double* e, const double* vel, double* F,
                             double* eF, const MeshView& m) {
  if (dir_y) {
    FLOW_LAUNCH2D(k_mass_energy_flux<1>, (ny + 1) - 2 * pad, nx - 2 * pad, nx,
                  ny, pad, dt, dt_h, rho, e, vel, F, eF, m.celldx, m.edgedx,
                  m.celldy, m.edgedy);
  } else {
    FLOW_LAUNCH2D(k_mass_energy_flux<0>, ny - 2 * pad, (nx + 1) - 2 * pad, nx,
                  ny, pad, dt, dt_h, rho, e, vel, F, eF, m.celldx, m.edgedx,
                  m.celldy, m.edgedy);
  }
}

void launch_mass_energy_update(cudaStream_t s, bool dir_y, int nx, int ny,
                               int pad, int first, double dt_h, double* rho,
                               const double* rho_old, double* e,
                               const double* F, const double* eF,
                               const MeshView& m) {
  if (dir_y) {
    FLOW_LAUNCH2D(k_mass_energy_update<1>, ny - 2 * pad, nx - 2 * pad, nx, ny,
                  pad, first, dt_h, rho, rho_old, e, F, eF, m.celldx, m.edgedx,
                  m.celldy, m.edgedy);
  } else {
    FLOW_LAUNCH2D(k_mass_energy_update<0>, ny - 2 * pad, nx - 2 * pad, nx, ny,
                  pad, first, dt_h, rho, rho_old, e, F, eF, m.celldx, m.edgedx,
                  m.celldy, m.edgedy);
  }
}

void launch_uF_x(cudaStream_t s, int nx, int ny, int pad, double dt_h,
                 const double* u, double* uF_x, const double* F_x,
                 const MeshView& m) {
  FLOW_LAUNCH2D(k_uF_x, ny - 2 * pad, nx - 2 * pad, nx, ny, pad, dt_h, u, uF_x,
                F_x, m.edgedx, m.edgedy, m.celldx);
}
void launch_uF_y(cudaStream_t s, int nx, int ny, int pad, double dt_h,
                 const double* u, const double* v, double* uF_y,
                 const double* F_y, const MeshView& m) {
  FLOW_LAUNCH2D(k_uF_y, (ny + 1) - 2 * pad, (nx + 1) - 2 * pad, nx, ny, pad,
                dt_h, u, v, uF_y, F_y, m.edgedx, m.edgedy, m.celldy);
}
void launch_vF_x(cudaStream_t s, int nx, int ny, int pad, double dt_h,
                 const double* u, const double* v, double* vF_x,
                 const double* F_x, const MeshView& m) {
  FLOW_LAUNCH2D(k_vF_x, (ny + 1) - 2 * pad, (nx + 1) - 2 * pad, nx, ny, pad,
                dt_h, u, v, vF_x, F_x, m.edgedx, m.celldy, m.celldx);
}
void launch_vF_y(cudaStream_t s, int nx, int ny, int pad, double dt_h,
                 const double* v, double* vF_y, const double* F_y,
                 const MeshView& m) {
  FLOW_LAUNCH2D(k_vF_y, ny - 2 * pad, nx - 2 * pad, nx, ny, pad, dt_h, v, vF_y,
                F_y, m.edgedy, m.celldx, m.celldy);
}

void launch_momentum_update(cudaStream_t s, int which, int nx, int ny, int pad,
                            double dt_h, int with_vel, double* mom, double* vel,
                            const double* flux, const double* rho,
                            const MeshView& m) {
  const int ru = ny - 2 * pad, cu = (nx + 1) - 2 * pad;
  const int rv = (ny + 1) - 2 * pad, cv = nx - 2 * pad;
#define FLOW_MU(K, R, C)                                                        \
  FLOW_LAUNCH2D(k_momentum_update<K>, R, C, nx, ny, pad, dt_h, with_vel, mom, \
                vel, flux, rho, m.edgedx, m.edgedy, m.celldx, m.celldy)
  switch (which) {
    case 0: FLOW_MU(0, ru, cu); break;
    case 1: FLOW_MU(1, ru, cu); break;
    case 2: FLOW_MU(2, rv, cv); break;
    default: FLOW_MU(3, rv, cv); break;
  }
#undef FLOW_MU
}

void launch_boundary(cudaStream_t s, int w, int h, int pad, double* arr,
                     int invert) {
  const long long n = 2LL * pad * w + 2LL * pad * (h - 2 * pad);
  if (n <= 0) return;
  const int threads = 256;
  launch_stage(k_boundary, dim3((unsigned)((n + threads - 1) / threads)), dim3(threads), s, w, h,
               pad, arr, invert == kInvertX, invert == kInvertY);
}

void launch_boundary2(cudaStream_t s, int w0, int h0, double* a0, int invert0, int w1, int h1,
                      double* a1, int invert1, int pad) {
  const long long n0 = 2LL * pad * w0 + 2LL * pad * (h0 - 2 * pad);
  const long long n1 = 2LL * pad * w1 + 2LL * pad * (h1 - 2 * pad);
  const long long n = n0 > n1 ? n0 : n1;
  if (n <= 0) return;
  const int threads = 256;
  launch_stage(k_boundary2, dim3((unsigned)((n + threads - 1) / threads), 2u), dim3(threads), s,
               w0, h0, a0, invert0 == kInvertX, invert0 == kInvertY, w1, h1, a1,
               invert1 == kInvertX, invert1 == kInvertY, pad);
}

void launch_copy(cudaStream_t s, size_t n, double* dst, const double* src) {
  if (n == 0) return;
  size_t blocks = (n + 255) / 256;
  if (blocks > 8192) blocks = 8192;
  launch_stage(k_copy, dim3((unsigned)blocks), dim3(256), s, n, dst, src);
}

}  // namespace flow
