// fused.cu -- the single-problem fused timestep (FP64 form behind
// solve_hydro_2d, and the mixed form gb300_mixed_solve): one kernel launch per
// phase, each CTA running one tile function of fused_tiles.cuh.
#include <array>
#include <cmath>
#include <cstddef>

#include "../../include/flow_gb300.h"
#include "fused.h"
#include "fused_tiles.cuh"
#include "lag_fused.cuh"
#include "profile.h"

namespace flow {
namespace {

using namespace tiles;

// Programmatic dependent launch: every kernel of the step is launched with
// programmatic stream serialisation, lets the next kernel launch as soon as
// all its own CTAs have started (pdl_trigger), and waits for the previous
// kernel to complete (its writes visible) before touching the state
// (pdl_wait).  The next kernel's CTAs thus take the SMs its predecessor's
// last wave leaves idle.  Outside such a launch both are no-ops.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" :::);
}

// The mesh test (mesh_test_part), the first kernel of a step: a block per part
// (one block alone took 1 us of a step longer on a 4096^2 mesh, whose 131 KB of
// spacings it read through one SM).  It also clears the CFL minimum slot and the
// block ticket for the step's Lagrangian kernels.  It does not let the pressure
// phase's blocks start early: while its own hold eight SMs they were spread
// unevenly, which the next kernels' blocks inherit (611x389 in motion: the
// viscosity phase 15.7 us for 11.4).
constexpr int kMeshThreads = 512;
__global__ void __launch_bounds__(kMeshThreads)
    k_mesh_test(int nx, int ny, const double* celldx, const double* edgedx, const double* celldy,
                const double* edgedy, double* ra, int known) {
  pdl_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *reinterpret_cast<unsigned long long*>(ra + kRaTicket) = 0ull;
    *reinterpret_cast<unsigned long long*>(ra + kRaMinBits) = ~0ull;
  }
  const unsigned r = mesh_test_part(nx, ny, celldx, edgedx, celldy, edgedy, ra + kRaMesh,
                                    (int)blockIdx.x, kMeshParts, known != 0);
  if (threadIdx.x == 0) {
    reinterpret_cast<unsigned char*>(ra + kRaMesh)[blockIdx.x] = (unsigned char)r;
  }
}

// How a kernel of the step runs: without flags (a mesh too small for them),
// with flags over its whole grid, or with flags over the listed tiles.  Two
// instantiations for the latter, as the tile of a block is uniform to the
// compiler only when it comes from blockIdx (the mixed form's pairs took 2%
// longer over a whole mesh with the choice made at run time).
enum : int { kNoFlags = 0, kWhole = 1, kListed = 2 };
template <int kMd, typename R>
__device__ __forceinline__ bool block_tile(const StepArgs<R>& a, int& bx, int& by) {
  if constexpr (kMd == kListed) {
    return listed_tile(a, (int)blockIdx.x, bx, by);
  } else {
    bx = blockIdx.x;
    by = blockIdx.y;
    return true;
  }
}

template <typename R, int kMd>
__global__ void __launch_bounds__(kCols, (Prec<R>::kMixed ? 0 : 8))
    k_lag_pressure(const StepArgs<R> a) {
  pdl_wait();
  pdl_trigger();
  // The phase's first block clears the block ticket (for the conservation totals
  // after the step), starts the CFL minimum from the tiles the step does not
  // visit, and clears what the second sweep's list blocks accumulate.
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    *reinterpret_cast<unsigned long long*>(a.ra + kRaTicket) = 0ull;
    *a.min_slot = a.from_rest_min ? *a.rest_min : ~0ull;
    if constexpr (kMd != kNoFlags) {
      *a.rest_min = ~0ull;
#pragma unroll
      for (int k = kRaTileCounts; k < kRaPartial; ++k) {
        *reinterpret_cast<unsigned long long*>(a.ra + k) = 0ull;
      }
    }
  }
  if constexpr (kMd == kListed) {
    // The skip marks this step leaves: set for every tile, those the first
    // sweep visits it writes itself.
    unsigned* marks = reinterpret_cast<unsigned*>(a.skipf);
    for (int q = blockIdx.x * kCols + threadIdx.x; q < a.skip_words; q += gridDim.x * kCols) {
      marks[q] = 0x01010101u;
    }
  }
  int bx, by;
  const bool uni = mesh_uniform<R>(a.mesh);
  if (block_tile<kMd>(a, bx, by)) {
    tile_lag_pressure<R, (kMd != kNoFlags), (kMd != kListed), (kMd != kListed)>(a, bx, by, uni);
  }
}
// With flags, the viscous-stress flags (a.qmask) are kept -- the viscosity
// kernel stores only warp rows with a non-zero stress, and the two kernels
// after it load only those.
template <typename R, int kMd>
__global__ void __launch_bounds__(kCols) k_lag_viscosity(const StepArgs<R> a) {
  pdl_wait();
  pdl_trigger();
  int bx, by;
  if (block_tile<kMd>(a, bx, by)) {
    tile_lag_viscosity<R, (kMd != kNoFlags), (kMd != kListed)>(a, bx, by);
  }
}
template <typename R, int kMd>
__global__ void __launch_bounds__(kCols) k_lag_viscous_accel(const StepArgs<R> a) {
  pdl_wait();
  pdl_trigger();
  int bx, by;
  const bool uni = mesh_uniform<R>(a.mesh);
  if (block_tile<kMd>(a, bx, by)) {
    tile_lag_viscous_accel<R, true, (kMd != kNoFlags)>(a, bx, by, uni);
  }
}
// Shock heating + CFL minimum (the first sweep applies the dt rule).
template <typename R, int kMd>
__global__ void __launch_bounds__(kCols) k_lag_energy_dt(const StepArgs<R> a) {
  __shared__ unsigned long long s_tile_min;  // the tile's CFL minimum (with flags)
  pdl_wait();
  pdl_trigger();
  int bx, by;
  constexpr bool kFlags = kMd != kNoFlags;
  const bool uni = mesh_uniform<R>(a.mesh);
  if (!block_tile<kMd>(a, bx, by)) return;
  tile_lag_energy_dt<R, true, kFlags, (kMd != kListed), (kMd != kListed)>(
      a, bx, by, uni, kFlags ? &s_tile_min : nullptr);
  // (Thread 0 wrote the minimum it stores here.)
  if (kFlags && a.cfl_tile && threadIdx.x == 0) {
    a.cfl_tile[(size_t)by * a.qm_stride + bx] = s_tile_min;
  }
}
// The first sweep's block 0 leaves the dt pair for the kernels after it.
template <typename R, bool kFirst>
__device__ __forceinline__ void store_dt(const StepArgs<R>& a) {
  if (kFirst && a.dt_from_min && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    const DtPair p = dt_rule(a, *a.min_slot);
    a.dt_slot[0] = p.dt;
    a.dt_slot[1] = p.dt_h;
  }
}
// ---------------------------------------------------------------------------
// Tile lists: the tiles the next step has to visit.  A cell in a tile the
// step's first sweep marked was at rest through the step (StepArgs::rest).  In
// the next step the flow reaches at most five cells past the cells that were
// not (one by the pressure jumps, one by the stresses, one by the sweeps'
// fluxes, two by the momentum fluxes), so a tile with every cell within
// kReach + pad of it marked (pad: the pressure phase's tiles start pad rows and
// columns earlier than the others') is left by every kernel of the next step
// as it is: it would test its flags and return.  On a blast that holds 1% of a
// 4096^2 mesh such tiles were half of a step (8192 tiles a kernel, 8 or so at
// once on an SM, about 2.5 us each).
constexpr int kListHeights = 4;               // tiles of 2, 4, 8 and 16 rows
constexpr int kListBand = 2 << (kListHeights - 1);
constexpr int kReach = 6;

struct ListArgs {
  int nx, ny, pad;
  const unsigned char* marks;  // this step's skip marks
  int mark_w, mark_tiles_x, mark_rows;
  int tx[2], bands;            // columns of 128- and 127-wide tiles, 16-row bands
  int blocks;                  // of each width (0: no lists)
  unsigned* list[2];           // [heights][tx * bands * 16 / height] each
  unsigned* counts;            // [2][kListHeights], cleared by the pressure phase
  // The CFL minimum over this step's shock-heating tiles that are not listed.
  const unsigned long long* cfl_tile;
  int cfl_tx, cfl_ty, cfl_rows;
  unsigned long long* rest_min;
};
// First entry of the list of height 2 << h in list[wide].
__host__ __device__ inline size_t list_offset(int tx, int bands, int h) {
  size_t o = 0;
  for (int k = 0; k < h; ++k) o += (size_t)tx * bands * (kListBand / (2 << k));
  return o;
}

// The lists, in blocks 0 .. 2 blocks - 1 of kCols threads: eight lanes per
// 16-row band of a tile column, each of which loads two or three bands of
// marks (all its loads in flight together) and decides one pair of rows.
__device__ __forceinline__ void tile_lists(const ListArgs& l, int block) {
  const int wd = block < l.blocks ? 0 : 1;  // the tile width
  const int t = (block - wd * l.blocks) * kCols + (int)threadIdx.x;
  constexpr int kSub = kListBand / 2;
  const int lane = threadIdx.x & 31, sub = lane & (kSub - 1), grp = lane & ~(kSub - 1);
  const int tx = l.tx[wd];
  const int k = t / kSub;
  const bool in = k < tx * l.bands;
  const int by = in ? k / tx : 0, bx = in ? k - by * tx : 0;
  const int pad = l.pad, D = kReach + pad;
  const int w = wd ? kCols - 1 : kCols;
  // The tile's columns and rows (clamped next to the walls: a ghost cell's
  // mirror source lies within pad of them) with the reach around them: three
  // columns of marks at most, where the ghost layers are no wider than 57.
  const int c0 = min(pad + bx * w, l.nx - 2 * pad);
  const int x0 = (max(c0 - D, pad) - pad) / l.mark_w;
  const int x1 = (min(c0 + w + D, l.nx - pad) - 1 - pad) / l.mark_w;
  const int r0 = pad + by * kListBand;
  const int lo = max(min(r0, l.ny - 2 * pad) - D, pad);
  const int hi = min(r0 + kListBand + D, l.ny - pad);
  const int b0 = (lo - pad) / l.mark_rows, b1 = (hi - 1 - pad) / l.mark_rows;
  // Bit b - b0: band b of marks holds a tile that was not at rest.
  unsigned long long moved = 0ull;
  constexpr int kRounds = 3;  // (kListBand + 2 D) / 2 + 1 bands at most, pad <= 4
  unsigned char m[kRounds][3];
#pragma unroll
  for (int q = 0; q < kRounds; ++q) {
    const int b = b0 + q * kSub + sub;
    const size_t row = (size_t)min(b, b1) * l.mark_tiles_x;
#pragma unroll
    for (int c = 0; c < 3; ++c) m[q][c] = l.marks[row + min(x0 + c, x1)];
  }
  for (int c = x0 + 3; c <= x1; ++c) {  // (wider ghost layers)
    for (int q = 0; q < kRounds; ++q) {
      m[q][0] &= l.marks[(size_t)min(b0 + q * kSub + sub, b1) * l.mark_tiles_x + c];
    }
  }
#pragma unroll
  for (int q = 0; q < kRounds; ++q) {
    const bool rest = (m[q][0] & m[q][1] & m[q][2]) != 0 || b0 + q * kSub + sub > b1;
    const unsigned v = __ballot_sync(0xffffffffu, in && !rest);
    moved |= (unsigned long long)((v >> grp) & ((1u << kSub) - 1)) << (q * kSub);
  }
  for (int q = kRounds * kSub; b0 + q <= b1; ++q) {  // (wide ghost layers)
    const size_t row = (size_t)(b0 + q) * l.mark_tiles_x;
    unsigned char rest = 1;
    for (int c = x0; c <= x1; ++c) rest &= l.marks[row + c];
    if (!rest) moved |= 1ull << min(q, 63);
  }
  const int s0 = r0 + 2 * sub;
  const int p0 = (max(min(s0, l.ny - 2 * pad) - D, pad) - pad) / l.mark_rows - b0;
  const int p1 = (min(s0 + 2 + D, l.ny - pad) - 1 - pad) / l.mark_rows - b0;
  const unsigned long long window =
      p0 > 63 ? 1ull << 63 : ((p1 >= 63 ? ~0ull : (1ull << (p1 + 1)) - 1) & ~((1ull << p0) - 1));
  // The tiles of height 2, then 4, 8 and 16: bit i of act, the group's i-th.
  unsigned act = (__ballot_sync(0xffffffffu, in && (moved & window) != 0ull) >> grp) &
                 ((1u << kSub) - 1);
  unsigned acts[kListHeights], all[kListHeights];
#pragma unroll
  for (int h = 0; h < kListHeights; ++h) {
    const int per = kSub >> h;
    if (h) {
      unsigned up = 0u;
      for (int i = 0; i < per; ++i) up |= ((act >> (2 * i)) & 3u) ? 1u << i : 0u;
      act = up;
    }
    acts[h] = act;
    all[h] = __ballot_sync(0xffffffffu, sub < per && ((act >> sub) & 1u));
  }
  // Lane h takes the warp's places in the list of height h (one round trip for
  // all of them).
  unsigned base = 0u;
#pragma unroll
  for (int h = 0; h < kListHeights; ++h) {
    if (lane == h) base = (unsigned)__popc(all[h]);
  }
  if (base) base = atomicAdd(l.counts + wd * kListHeights + lane, base);
#pragma unroll
  for (int h = 0; h < kListHeights; ++h) {
    const int per = kSub >> h;
    const bool mine = sub < per && ((acts[h] >> sub) & 1u);
    const unsigned at = __shfl_sync(0xffffffffu, base, h) + __popc(all[h] & ((1u << lane) - 1));
    if (mine) {
      l.list[wd][list_offset(tx, l.bands, h) + at] =
          ((unsigned)(by * per + sub) << 16) | (unsigned)bx;
    }
    if (wd == 0 && l.cfl_rows == (2 << h)) {
      const int ty = by * per + sub;
      unsigned long long c = ~0ull;
      if (in && sub < per && !mine && bx < l.cfl_tx && ty < l.cfl_ty) {
        c = l.cfl_tile[(size_t)ty * l.cfl_tx + bx];
      }
      c = warp_min_u64(c);
      if (lane == 0 && c != ~0ull) atomicMin(l.rest_min, c);
    }
  }
}

// Momentum pairs (flux fused with its update): x pairs share a row's fluxes
// through shared memory (127 faces per CTA), y pairs march down columns.
// Tile k of a 1-D launch.
template <int kMd, typename R>
__device__ __forceinline__ bool line_tile(const StepArgs<R>& a, int k, int& bx, int& by) {
  if constexpr (kMd == kListed) {
    return listed_tile(a, k, bx, by);
  } else {
    by = k / a.grid_x;
    bx = k - by * a.grid_x;
    return true;
  }
}
// With flags, the mass-flux flags (a.fxflag, a.fyflag) are kept -- the sweeps
// store only warps with a non-zero mass flux, and the momentum pairs load only
// those.
// kLists (a second sweep): the last 2 l.blocks blocks of the (1-D) launch form
// the next step's tile lists beside the sweep, which changes neither the marks
// nor the minima they are formed from; as a kernel of their own the lists took 7
// to 20 us a step, and beside the step's last launch, which is short, 5.
template <typename R, bool kFirst, int kMd, bool kLists>
__global__ void __launch_bounds__(kCols, Prec<R>::kMixed ? 8 : 7) k_mass_sweep_x(
    const StepArgs<R> a, const SweepArgs<R> s, const ListArgs l) {
  pdl_wait();
  pdl_trigger();
  int bx, by;
  const bool uni = mesh_uniform<R>(a.mesh);
  if constexpr (kLists) {
    const int n = (int)gridDim.x - 2 * l.blocks;
    if ((int)blockIdx.x >= n) {
      tile_lists(l, (int)blockIdx.x - n);
      return;
    }
  }
  if (kLists ? line_tile<kMd>(a, blockIdx.x, bx, by) : block_tile<kMd>(a, bx, by)) {
    tile_mass_sweep_x<R, kFirst, true, (kMd != kNoFlags), (kMd != kListed)>(a, s, bx, by, uni);
  }
  store_dt<R, kFirst>(a);
}
template <typename R, bool kFirst, int kMd, bool kLists>
__global__ void __launch_bounds__(kCols, Prec<R>::kMixed ? 7 : 6) k_mass_sweep_y(
    const StepArgs<R> a, const SweepArgs<R> s, const ListArgs l) {
  pdl_wait();
  pdl_trigger();
  int bx, by;
  const bool uni = mesh_uniform<R>(a.mesh);
  if constexpr (kLists) {
    const int n = (int)gridDim.x - 2 * l.blocks;
    if ((int)blockIdx.x >= n) {
      tile_lists(l, (int)blockIdx.x - n);
      return;
    }
  }
  if (kLists ? line_tile<kMd>(a, blockIdx.x, bx, by) : block_tile<kMd>(a, bx, by)) {
    tile_mass_sweep_y<R, kFirst, true, (kMd != kNoFlags), (kMd != kListed)>(a, s, bx, by, uni);
  }
  store_dt<R, kFirst>(a);
}
// One launch runs one pair, or two that do not read what the other writes
// (launch_step): two dependent launches of a few microseconds each become one.
enum : int { kNone = 0, kXU = 1, kXV = 2, kYU = 3, kYV = 4 };  // direction and momentum
template <typename R, int kPair, bool kVel, int kMd>
__device__ __forceinline__ void pair_tile(const StepArgs<R>& a, int bx, int by, bool uni) {
  constexpr bool kFl = kMd != kNoFlags, kTest = kMd != kListed;
  if constexpr (kPair == kXU) tile_mom_x<R, false, kVel, true, kFl, kTest, kTest>(a, bx, by, uni);
  else if constexpr (kPair == kXV)
    tile_mom_x<R, true, kVel, true, kFl, kTest, kTest>(a, bx, by, uni);
  else if constexpr (kPair == kYU)
    tile_mom_y<R, false, kVel, true, kFl, kTest, kTest>(a, bx, by, uni);
  else if constexpr (kPair == kYV)
    tile_mom_y<R, true, kVel, true, kFl, kTest, kTest>(a, bx, by, uni);
}
// The tiles of pair A (blocks 0 .. na - 1), then those of pair B.
// (Two FP64 velocity pairs: six CTAs an SM; left to itself the compiler takes 86
// registers, which hold five -- 253 us for 244 at 2048x2048 in motion.)
template <typename R, int kA, bool kVelA, int kB, bool kVelB, int kMd>
__global__ void __launch_bounds__(kCols, (kVelA && kVelB && !Prec<R>::kMixed ? 6 : 0))
    k_mom(const StepArgs<R> a, const StepArgs<R> b, int na) {
  pdl_wait();
  pdl_trigger();
  const bool uni = mesh_uniform<R>(a.mesh);
  const int k = (int)blockIdx.x;
  int bx, by;
  if constexpr (kB != kNone) {
    if (k >= na) {
      if (line_tile<kMd>(b, k - na, bx, by)) pair_tile<R, kB, kVelB, kMd>(b, bx, by, uni);
      return;
    }
  }
  if (line_tile<kMd>(a, k, bx, by)) pair_tile<R, kA, kVelA, kMd>(a, bx, by, uni);
}

// The whole Lagrangian phase of the FP64 step in one kernel (lag_fused.cuh):
// pressure, viscosity, viscous acceleration, shock heating and the CFL
// minimum; the last block to finish (ticket in reduce_array) applies the dt
// rule.  A tile whose row copies were lost records GB300_ERR_TIMEOUT in the
// status word and leaves the dt pair unchanged.
__global__ void __launch_bounds__(lagf::kT, 4) k_lag_fused(const lagf::LagArgs a) {
  __shared__ lagf::LagSmem sm;
  __shared__ unsigned long long s_warp[lagf::kWarps];
  __shared__ bool s_last;
  pdl_wait();
  pdl_trigger();
  lagf::CflBest cfl;
  const bool uniform = mesh_uniform<double>(a.mesh);
  const bool ok = uniform
                      ? lagf::lag_tile<true>(a, sm, blockIdx.x, blockIdx.y, cfl)
                      : lagf::lag_tile<false>(a, sm, blockIdx.x, blockIdx.y, cfl);
  if (!ok) {
    if (threadIdx.x == 0) {
      atomicExch(reinterpret_cast<unsigned long long*>(a.ra + kRaStatus),
                 (unsigned long long)GB300_ERR_TIMEOUT);
    }
    return;
  }
  unsigned long long best = ~0ull;
  if (cfl.kbest >= 0) best = (unsigned long long)dbits(cfl.c_best * d_rsqrt(cfl.s_best));
  if (uniform) {
    const UniformMesh um = uniform_mesh(a.mesh);
    best = cfl.max.candidate(um.dx, um.dy);
  }
  best = warp_min_u64(best);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long b = s_warp[0];
    for (int w = 1; w < lagf::kWarps; ++w) b = (s_warp[w] < b) ? s_warp[w] : b;
    atomicMin(a.min_slot, b);
    __threadfence();
    unsigned long long* ticket = reinterpret_cast<unsigned long long*>(a.ra + kRaTicket);
    s_last = (atomicAdd(ticket, 1ull) == (unsigned long long)gridDim.x * gridDim.y - 1);
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    // The leapfrog dt/dt_h rule of omp3/flow.c:103-105 (finish_dt).
    const unsigned long long gmin = atomicExch(a.min_slot, ~0ull);
    const double cflv = d_min_pos(a.max_dt, dfrom((long long)gmin));
    const double limited = dmin(cflv, __dmul_rn(FLOW_C_M, a.dt_h));
    const double dt = __dmul_rn(0.5, __dadd_rn(__dmul_rn(kCT, limited), a.dt_h));
    a.dt_slot[0] = dt;
    a.dt_slot[1] = a.first_step ? dt : __dmul_rn(kCT, limited);
    *reinterpret_cast<unsigned long long*>(a.ra + kRaTicket) = 0ull;
  }
}

// Copies the changed energies (with their ghost images) and momenta of the
// fused Lagrangian kernel into the state arrays.  Each thread reads the three
// change masks of one (mask row, tile) pair -- 48 contiguous bytes, so the
// scan is one coalesced pass over the masks -- and the warp then copies the
// flagged values of each non-empty pair together, one lane per column.
constexpr int kApplyThreads = 256;
__global__ void __launch_bounds__(kApplyThreads)
    k_lag_apply(const lagf::LagArgs a, double* e, double* rho_u, double* rho_v) {
  pdl_wait();
  pdl_trigger();
  const int nx = a.nx, ny = a.ny, pad = a.pad;
  const int lane = threadIdx.x & 31;
  const int pairs = (ny + 1) * a.ntx;
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < pairs; base += stride) {
    const int k = base + (int)threadIdx.x;
    uint4 m[lagf::kMaskFields] = {};
    bool any = false;
    if (k < pairs) {
      const int row = k / a.ntx;
      // Mask rows the tiles write: cells and x faces pad .. ny-pad-1, y faces
      // pad .. ny-pad.
      if (row >= pad && row <= ny - pad) {
        const uint4* mk = reinterpret_cast<const uint4*>(a.masks) + (size_t)k * lagf::kMaskFields;
#pragma unroll
        for (int f = 0; f < lagf::kMaskFields; ++f) {
          if (f != lagf::kMaskRhoV && row == ny - pad) continue;
          m[f] = mk[f];
          any |= (m[f].x | m[f].y | m[f].z | m[f].w) != 0u;
        }
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, any);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const int kk = __shfl_sync(0xffffffffu, k, src);
      const int row = kk / a.ntx;
      const int c0 = pad + (kk - row * a.ntx) * lagf::kW - lagf::kHalo;
#pragma unroll
      for (int f = 0; f < lagf::kMaskFields; ++f) {
        const unsigned w0 = __shfl_sync(0xffffffffu, m[f].x, src);
        const unsigned w1 = __shfl_sync(0xffffffffu, m[f].y, src);
        const unsigned w2 = __shfl_sync(0xffffffffu, m[f].z, src);
        const unsigned w3 = __shfl_sync(0xffffffffu, m[f].w, src);
        const unsigned words[lagf::kWarps] = {w0, w1, w2, w3};
#pragma unroll
        for (int w = 0; w < lagf::kWarps; ++w) {
          if (!((words[w] >> lane) & 1u)) continue;
          const int col = c0 + 32 * w + lane;
          if (f == lagf::kMaskE) {
            const size_t ci = cidx(nx, row, col);
            const double val = a.e_new[ci];
            e[ci] = val;
            mirror(true, e, nx, ny, pad, row, col, val, false, false);
          } else if (f == lagf::kMaskRhoU) {
            const size_t fi = fidx(nx, row, col);
            rho_u[fi] = a.rho_u_new[fi];
          } else {
            const size_t ci = cidx(nx, row, col);
            rho_v[ci] = a.rho_v_new[ci];
          }
        }
      }
    }
  }
}

// Launches kernel k with programmatic stream serialisation (see pdl_wait).
template <typename... KArgs, typename... Args>
void launch_pdl_block(void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t s,
                      Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
  count_launches(1);
}
template <typename... KArgs, typename... Args>
void launch_pdl(void (*k)(KArgs...), dim3 grid, cudaStream_t s, Args... args) {
  launch_pdl_block(k, grid, dim3(kCols), s, args...);
}

// The previous step's tile lists, by tile width (128, 127) and height.
struct TileLists {
  bool use = false;
  const unsigned* list[2][kListHeights] = {};
  int n[2][kListHeights] = {};
};
inline int height_index(int rows) { return rows == 2 ? 0 : rows == 4 ? 1 : rows == 8 ? 2 : 3; }
// The grid of a kernel over the tiles of `full` (set in a): all of them, or
// the listed ones.
template <typename R>
dim3 tile_grid(StepArgs<R>& a, const TileLists& tl, int narrow, dim3 full) {
  a.grid_x = (int)full.x;
  a.grid_y = (int)full.y;
  if (!tl.use) {
    a.tiles = nullptr;
    return full;
  }
  const int h = height_index(a.rows);
  a.tiles = tl.list[narrow][h];
  a.n_tiles = tl.n[narrow][h];
  return dim3((unsigned)(a.n_tiles > 0 ? a.n_tiles : 1));
}

inline dim3 strip_grid(int cols, int rows, int tile_rows, int cols_per_cta = kCols) {
  return dim3((unsigned)((cols + cols_per_cta - 1) / cols_per_cta),
              (unsigned)((rows + tile_rows - 1) / tile_rows));
}

// Tile heights of a step, by kernel.  A warp's FP64 instructions issue one per
// 64 clocks, and depend on one another at that distance too, so a tile takes
// its rows one after another at about 1 to 3 us a row, and a kernel whose tiles
// fit the SMs at once takes as long as its longest tile: on a 48x32 mesh
// 16-row tiles made a step of 345 us with most SMs idle.  The height taken is
// the one with the least time on the busiest SM,
//   (rows + kHaloRows) * max(ceil(tiles / SMs), tiles that an SM overlaps):
// kHaloRows for a tile's first face flux, table set-up and first loads (about
// a row's time or two); an SM overlaps the tiles whose latencies hide behind
// one another's, three in the FP64 form (a third of a row's time is FP64
// issue), six in the mixed form.
struct StepRows {
  int lag = 16, energy = 16, accel = 16, sweep = 16, mom_vel = 16, mom_flux = 16;
};
// Shortest tiles: with flags, the second sweep's skip test reads the marks one
// band either side of its own, which hold the two rows it reaches past it.
constexpr int kMinRowsFlags = 2;
constexpr int kMaxRowsStep = 16;
// The shock-heating tiles keep their minima from step to step by tile, so a
// new height makes that kernel visit the whole mesh once.  It starts at eight
// rows at most (a run's first step does not know what moves) and stays there
// while the lists are in use.
constexpr int kRowsEnergy = 8;
// The viscous update and the momentum pairs without a velocity update leave
// tiles without a stress or a mass flux at once, so their longest chain of
// rows bounds them (4096x2048 moving everywhere: the viscous update takes
// 196 us with 16 rows, 181 with 8; 2048^2 mixed: a step 556 us, 546 with 8).
constexpr int kRowsSparse = 8;
constexpr double kHaloRows = 1.5, kOverlap64 = 3.0, kOverlapMixed = 6.0;
inline double rows_cost(double tiles, int rows, double overlap) {
  const double per_sm = ceil(tiles / num_sms());
  return (rows + kHaloRows) * (per_sm > overlap ? per_sm : overlap);
}
// The tiles of each height a step visits: all of a mesh of cols x rows, or
// counts of the lists (index: height 2 << i).  was: the previous step's
// height, kept unless another is a fifth cheaper (0: none).
int pick_rows(int cols, int rows, int cols_per_cta, const unsigned* counts, int min_rows,
              int was, double overlap) {
  const double tx = (cols + cols_per_cta - 1) / cols_per_cta;
  auto cost = [&](int h) {
    return rows_cost(counts ? (double)counts[height_index(h)] : tx * ((rows + h - 1) / h), h,
                     overlap);
  };
  int best = kMaxRowsStep;
  for (int h = kMaxRowsStep / 2; h >= min_rows; h /= 2) {
    if (cost(h) < cost(best)) best = h;
  }
  return was >= min_rows && cost(best) > 0.8 * cost(was) ? was : best;
}
// counts: the lengths of the tile lists ([2][kListHeights]), or null where
// the step visits every tile; was: the step before, when this one follows it.
StepRows pick_step_rows(int nx, int ny, int pad, const unsigned* counts, bool flags,
                        const StepRows* was, double overlap) {
  const int w = nx - 2 * pad, h = ny - 2 * pad;
  const int lo = flags ? kMinRowsFlags : 1;
  const unsigned* narrow = counts ? counts + kListHeights : nullptr;
  StepRows r;
  r.lag = pick_rows(w, h, kCols, counts, lo, was ? was->lag : 0, overlap);
  r.accel = r.lag > kRowsSparse ? kRowsSparse : r.lag;
  r.energy = r.lag;
  if (flags && counts) {
    r.energy = was->energy <= kRowsEnergy ? was->energy : kRowsEnergy;
  } else if (flags && !was && r.energy > kRowsEnergy) {
    r.energy = kRowsEnergy;
  }
  r.sweep = pick_rows(w + 1, h, kCols - 1, narrow, lo, was ? was->sweep : 0, overlap);
  r.mom_vel = r.sweep;
  r.mom_flux = r.sweep > kRowsSparse ? kRowsSparse : r.sweep;
  return r;
}
template <typename R>
StepArgs<R> with_rows(const StepArgs<R>& a, int rows) {
  StepArgs<R> b = a;
  b.rows = rows;
  return b;
}

// x pair for rho_u (kV false): x-faces pad .. nx-pad, 127 per CTA; for rho_v:
// y-faces pad .. nx-pad-1.  Rows: the faces' rows.
// Launches the instantiation of kernel template K (its arguments before the
// mode and after it) that a step runs.
#define FLOW_LAUNCH_MODE(md, g, s, args, K, ...)                                       \
  do {                                                                                 \
    if ((md) == kNoFlags) launch_pdl(K<__VA_ARGS__, kNoFlags>, g, s, FLOW_UNPACK args); \
    else if ((md) == kWhole) launch_pdl(K<__VA_ARGS__, kWhole>, g, s, FLOW_UNPACK args); \
    else launch_pdl(K<__VA_ARGS__, kListed>, g, s, FLOW_UNPACK args);                  \
  } while (0)
#define FLOW_UNPACK(...) __VA_ARGS__
template <typename R>
int step_mode(const StepArgs<R>& a) {
  return !a.qmask ? kNoFlags : a.tiles ? kListed : kWhole;
}

// The tiles of one momentum pair: x pairs have 127 faces per CTA; rho_u lives
// on x-faces pad .. nx-pad, rho_v on y-faces pad .. nx-pad-1 of one more row.
template <typename R, int kPair, bool kVel>
StepArgs<R> pair_args(const StepArgs<R>& a0, const StepRows& sr, const TileLists& tl, int& tiles) {
  constexpr bool kV = kPair == kXV || kPair == kYV, kX = kPair == kXU || kPair == kXV;
  StepArgs<R> a = with_rows(a0, kVel ? sr.mom_vel : sr.mom_flux);
  const int cols = kV ? (a.nx - 2 * a.pad) : (a.nx + 1 - 2 * a.pad);
  const int rows = kV ? (a.ny + 1 - 2 * a.pad) : (a.ny - 2 * a.pad);
  const dim3 g =
      tile_grid(a, tl, kX ? 1 : 0, strip_grid(cols, rows, a.rows, kX ? kCols - 1 : kCols));
  tiles = (int)(g.x * g.y);
  return a;
}
template <typename R, int kA, bool kVelA, int kB, bool kVelB>
void launch_mom(cudaStream_t s, const StepArgs<R>& a0, const StepRows& sr, const TileLists& tl) {
  int na = 0, nb = 0;
  const StepArgs<R> a = pair_args<R, kA, kVelA>(a0, sr, tl, na);
  const StepArgs<R> b = pair_args<R, kB, kVelB>(a0, sr, tl, nb);
  if (kB == kNone) nb = 0;
  const dim3 g((unsigned)(na + nb));
  const int md = step_mode(a);
  if (md == kNoFlags) launch_pdl(k_mom<R, kA, kVelA, kB, kVelB, kNoFlags>, g, s, a, b, na);
  else if (md == kWhole) launch_pdl(k_mom<R, kA, kVelA, kB, kVelB, kWhole>, g, s, a, b, na);
  else launch_pdl(k_mom<R, kA, kVelA, kB, kVelB, kListed>, g, s, a, b, na);
}

// lists: formed beside the step's second sweep (blocks 0: none).
template <typename R, bool kY>
void launch_sweep(cudaStream_t s, const StepArgs<R>& a0, bool first, const SweepArgs<R>& sw,
                  const TileLists& tl, const ListArgs& lists) {
  StepArgs<R> a = a0;
  const int pad = a.pad;
  // The x sweep: faces pad .. nx-pad; every CTA advances 127 columns.
  const dim3 g = tile_grid(a, tl, kY ? 0 : 1,
                           kY ? strip_grid(a.nx - 2 * pad, a.ny - 2 * pad, a.rows)
                              : strip_grid(a.nx + 1 - 2 * pad, a.ny - 2 * pad, a.rows, kCols - 1));
  const int md = step_mode(a);
#define FLOW_SWEEP(FIRST, MODE, LISTS, GRID)                                                  \
  do {                                                                                        \
    if constexpr (kY) launch_pdl(k_mass_sweep_y<R, FIRST, MODE, LISTS>, GRID, s, a, sw, lists); \
    else launch_pdl(k_mass_sweep_x<R, FIRST, MODE, LISTS>, GRID, s, a, sw, lists);            \
  } while (0)
  if (first) {
    if (md == kNoFlags) FLOW_SWEEP(true, kNoFlags, false, g);
    else if (md == kWhole) FLOW_SWEEP(true, kWhole, false, g);
    else FLOW_SWEEP(true, kListed, false, g);
  } else if (lists.blocks) {
    const dim3 line(g.x * g.y + 2 * (unsigned)lists.blocks);
    if (md == kListed) FLOW_SWEEP(false, kListed, true, line);
    else FLOW_SWEEP(false, kWhole, true, line);
  } else {
    if (md == kNoFlags) FLOW_SWEEP(false, kNoFlags, false, g);
    else if (md == kWhole) FLOW_SWEEP(false, kWhole, false, g);
    else FLOW_SWEEP(false, kListed, false, g);
  }
#undef FLOW_SWEEP
}
template <typename R>
void launch_mass(cudaStream_t s, const StepArgs<R>& a, bool dir_y, bool first,
                 const SweepArgs<R>& sw, const TileLists& tl, const ListArgs& lists) {
  if (dir_y) launch_sweep<R, true>(s, a, first, sw, tl, lists);
  else launch_sweep<R, false>(s, a, first, sw, tl, lists);
}

// Blocks of k_lag_apply: one thread per (mask row, tile) pair, at most 8
// blocks per SM (a grid-stride loop covers the rest).
inline int apply_blocks(const lagf::LagArgs& l) {
  const int pairs = (l.ny + 1) * l.ntx;
  const int need = (pairs + kApplyThreads - 1) / kApplyThreads;
  return need < 8 * num_sms() ? need : 8 * num_sms();
}

// One timestep of either form; first/second are the two mass sweeps' buffers.
// lag: the FP64 form's one-kernel Lagrangian phase (k_lag_fused +
// k_lag_apply), or null for the four separate Lagrangian kernels.
template <typename R>
void launch_step(cudaStream_t s, const StepArgs<R>& a, int tt,
                 const SweepArgs<R>& first, const SweepArgs<R>& second,
                 StepProfiler& prof, const StepRows& sr,
                 const TileLists& tl, const ListArgs& lists,
                 const lagf::LagArgs* lag = nullptr) {
  const int nx = a.nx, ny = a.ny, pad = a.pad;
  // The whole-mesh spacing test the tiles read, formed by every step: the
  // caller may have written the spacing arrays since the last.  (A launch more,
  // 1 to 2 us of a step: 611x389 in motion 217.5 -> 219 us, a box on 1024^2 with
  // the totals 137 -> 138.5, a blast on 4096^2 136 -> 137.5.)
  prof.mark("mesh_test");
  launch_pdl_block(k_mesh_test, dim3(kMeshParts), dim3(kMeshThreads), s, nx, ny, a.celldx, a.edgedx,
                   a.celldy, a.edgedy, a.ra, a.rest != nullptr ? 1 : 0);
  if (lag) {
    const int nty = (ny - 2 * pad + lag->rows - 1) / lag->rows;
    prof.mark("lag_fused");
    launch_pdl_block(k_lag_fused, dim3((unsigned)lag->ntx, (unsigned)nty), dim3(lagf::kT), s,
                     *lag);
    prof.mark("lag_apply");
    launch_pdl_block(k_lag_apply, dim3((unsigned)apply_blocks(*lag)), dim3(kApplyThreads), s,
                     *lag, const_cast<double*>(lag->e), const_cast<double*>(lag->rho_u),
                     const_cast<double*>(lag->rho_v));
  } else {
    prof.mark("lag_pressure");
    StepArgs<R> al = a;
    dim3 g = tile_grid(al, tl, 0, strip_grid(nx, ny, a.rows));
    FLOW_LAUNCH_MODE(step_mode(al), g, s, (al), k_lag_pressure, R);
    prof.mark("lag_viscosity");
    g = tile_grid(al, tl, 0, strip_grid(nx - 2 * pad, ny - 2 * pad, a.rows));
    FLOW_LAUNCH_MODE(step_mode(al), g, s, (al), k_lag_viscosity, R);
    prof.mark("lag_viscous_accel");
    StepArgs<R> aa = with_rows(a, sr.accel);
    g = tile_grid(aa, tl, 0, strip_grid(nx + 1 - 2 * pad, ny + 1 - 2 * pad, aa.rows));
    FLOW_LAUNCH_MODE(step_mode(aa), g, s, (aa), k_lag_viscous_accel, R);
    prof.mark("lag_energy_dt");
    // (All tiles where the minima of those off the list are not known.)
    StepArgs<R> ae = with_rows(a, sr.energy);
    g = tile_grid(ae, a.cfl_known ? tl : TileLists{}, 0,
                  strip_grid(nx - 2 * pad, ny - 2 * pad, ae.rows));
    FLOW_LAUNCH_MODE(step_mode(ae), g, s, (ae), k_lag_energy_dt, R);
  }

  // The advection phase reads velocity flags only when this step's
  // Lagrangian kernels wrote them (not the one-kernel phase).
  StepArgs<R> ad = a;
  if (lag) {
    ad.vflag = nullptr;
    ad.dt_from_min = 0;  // (its last block has applied the dt rule)
  }
  const StepArgs<R> as = with_rows(ad, sr.sweep);
  const bool x_first = (tt % 2 == 0);
  // With flags, the first sweep marks the tiles it skips (in its own grid);
  // the second reads their cells from the first sweep's input.
  SweepArgs<R> sw1 = first, sw2 = second;
  if (a.skipf) {
    sw1.skip = sw2.skip = a.skipf;
    sw1.skip_tiles_x = sw2.skip_tiles_x = x_first ? a.fx_stride / 4 : a.qm_stride;
    sw1.skip_bands = sw2.skip_bands = (ny - 2 * pad + sr.sweep - 1) / sr.sweep;
    sw2.r_alt = first.r_in;
    sw2.e_alt = first.e_in;
    sw2.r_alt_r = first.r_in_r;
    sw2.e_alt_r = first.e_in_r;
  }
  prof.mark(x_first ? "mass_sweep_x" : "mass_sweep_y");
  launch_mass(s, as, !x_first, true, sw1, tl, lists);
  prof.mark(x_first ? "mass_sweep_y" : "mass_sweep_x");
  launch_mass(s, as, x_first, false, sw2, tl, lists);

  // Momentum: each flux fused with its update, in the reference order; the
  // pair that recomputes a velocity comes first in each chain.  Two pairs share
  // a launch where neither reads what the other writes: the y pairs take the
  // Lagrangian velocities as their wind, so both velocity pairs of an even
  // step, whose flux pairs then read only the advected velocities; of an odd
  // step the y flux pair of rho_u and the x velocity pair of rho_v.
  if (tt % 2) {
    prof.mark("mom_uFx");
    launch_mom<R, kXU, true, kNone, false>(s, ad, sr, tl);
    prof.mark("mom_uFy_vFx");
    launch_mom<R, kYU, false, kXV, true>(s, ad, sr, tl);
    prof.mark("mom_vFy");
    launch_mom<R, kYV, false, kNone, false>(s, ad, sr, tl);
  } else {
    prof.mark("mom_uFy_vFy");
    launch_mom<R, kYU, true, kYV, true>(s, ad, sr, tl);
    prof.mark("mom_uFx_vFx");
    launch_mom<R, kXU, false, kXV, false>(s, ad, sr, tl);
  }
}

// Copies the step's header (reduce_array before the partials) to page-locked
// host memory.
__global__ void k_step_head(const double* ra, double* host) {
  pdl_wait();
  if (threadIdx.x < kRaPartial) host[threadIdx.x] = ra[threadIdx.x];
}

int finish_step(cudaStream_t s, Mesh* mesh, double* ra, StepProfiler& prof,
                const char* where, unsigned* counts) {
  // dt, dt_h (slots 0, 1), the status word (slot 5) and the lengths of the
  // tile lists (slots 13 .. 16) at once.
  double local[kRaPartial];
  double* head = pinned_head();
  if (head) launch_pdl_block(k_step_head, dim3(1), dim3(32), s, ra, head);
  {
    const int st = check_launch(where);
    if (st != GB300_OK) return st;
  }
  if (!head) {
    head = local;
    cudaMemcpyAsync(head, ra + kRaDt, sizeof(local), cudaMemcpyDeviceToHost, s);
  }
  const cudaError_t err = cudaStreamSynchronize(s);
  if (err != cudaSuccess) {
    return record_error(GB300_ERR_CUDA, "%s: %s", where, cudaGetErrorString(err));
  }
  prof.end();
  unsigned long long status;
  memcpy(&status, &head[kRaStatus], sizeof(status));
  if (status != 0ull) {
    cudaMemsetAsync(ra + kRaStatus, 0, sizeof(double), s);
    return record_error(GB300_ERR_TIMEOUT,
                        "%s: a row copy of the Lagrangian kernel did not arrive", where);
  }
  memcpy(counts, &head[kRaTileCounts], 2 * kListHeights * sizeof(unsigned));
  const double pair[2] = {head[kRaDt], head[kRaDtH]};
  mesh->dt = pair[0];
  mesh->dt_h = pair[1];
  return GB300_OK;
}

// Where the fused step's flags sit in reduce_array after the reduction
// partials (ra + kRaQFlags), when it holds them (it has nx*ny doubles, as the
// arch layer allocates it); a mesh too small for them stores and reads every
// stress and flux.  Offsets in 4-byte words: the per-tile CFL minima (two
// words per shock-heating tile) and the conservation totals' tile partials
// (four words per tile) first, 8-byte aligned; then the stress
// flags ((ny - 2 pad) x stride words), the y mass-flux flags
// ((ny + 1 - 2 pad) x stride), the x mass-flux flags ((ny - 2 pad) x xtiles),
// the velocity flags (ny x vtiles) and the skip marks of even and odd steps
// (a step's first sweep writes its own half; the next step reads it while its
// own first sweep writes the other), and the tile lists that even and odd steps
// leave (the step's last kernel forms its own while it reads the previous
// step's).
// Conservation tiles: 128 columns and the fewest rows, 16 times a power of two,
// that leave at most kConsTiles of them.  128 rows a tile kept a 1024^2 mesh's
// 64 blocks at their chain of loads and additions for 30 us; shorter tiles
// spread it, and the last block adds at most 32 partials a thread.
constexpr int kConsTile = 128, kConsTiles = 4096;
inline int cons_rows(int cols, long long rows) {
  const long long tx = (cols + kConsTile - 1) / kConsTile;
  int h = 16;
  while (tx * ((rows + h - 1) / h) > kConsTiles && h < (1 << 20)) h *= 2;
  return h;
}
struct FlagLayout {
  bool fits = false;
  int stride = 0, xtiles = 0, vtiles = 0, cons_tx = 0, cons_ty = 0, cons_h = 0;
  int list_tx[2] = {0, 0}, list_bands = 0;
  size_t cfl = 0, cons = 0, q = 0, fy = 0, fx = 0, v = 0, marks = 0, sk_words = 0, lists = 0,
         list_words[2] = {0, 0};
};
FlagLayout flag_layout(int nx, int ny, int pad) {
  FlagLayout L;
  L.stride = (nx - 2 * pad + kCols - 1) / kCols;
  L.xtiles = (nx + 1 - 2 * pad + kCols - 2) / (kCols - 1);
  L.vtiles = (nx + kCols - 1) / kCols;
  const long long rows = ny - 2 * pad;
  if (L.stride <= 0 || rows <= 0) return L;
  L.cons_tx = (nx - 2 * pad + kConsTile - 1) / kConsTile;
  L.cons_h = cons_rows(nx - 2 * pad, rows);
  L.cons_ty = (int)((rows + L.cons_h - 1) / L.cons_h);
  const long long bands = (rows + kMinRowsFlags - 1) / kMinRowsFlags;  // tile bands, at most
  L.sk_words = ((size_t)bands * (L.xtiles > L.stride ? L.xtiles : L.stride) + 3) / 4;
  L.cfl = 0;
  L.cons = L.cfl + 2 * (size_t)bands * L.stride;
  L.q = L.cons + 4 * (size_t)L.cons_tx * L.cons_ty;
  L.fy = L.q + (size_t)rows * L.stride;
  L.fx = L.fy + (size_t)(rows + 1) * L.stride;
  L.v = L.fx + (size_t)rows * L.xtiles;
  L.marks = L.v + (size_t)ny * L.vtiles;
  L.lists = L.marks + 2 * L.sk_words;
  L.list_tx[0] = L.vtiles;
  L.list_tx[1] = L.xtiles;
  L.list_bands = (ny + kListBand - 1) / kListBand;
  for (int w = 0; w < 2; ++w) {
    L.list_words[w] = list_offset(L.list_tx[w], L.list_bands, kListHeights);
  }
  const size_t words = L.lists + 2 * (L.list_words[0] + L.list_words[1]);
  L.fits = (size_t)kRaQFlags * sizeof(double) + words * sizeof(unsigned) <=
           (size_t)nx * ny * sizeof(double);
  return L;
}

template <typename R>
void fill_mesh_args(StepArgs<R>& a, const Mesh* mesh, int tt, double* ra) {
  a.nx = mesh->local_nx;
  a.ny = mesh->local_ny;
  a.pad = mesh->pad;
  a.edgedx = mesh->edgedx;
  a.edgedy = mesh->edgedy;
  a.celldx = mesh->celldx;
  a.celldy = mesh->celldy;
  a.ra = ra;
  a.min_slot = reinterpret_cast<unsigned long long*>(ra + kRaMinBits);
  a.mesh = ra + kRaMesh;
  a.dt_slot = ra + kRaDt;
  a.dt = mesh->dt;
  a.dt_h = mesh->dt_h;
  a.max_dt = mesh->max_dt;
  a.first_step = (tt == 0);
  a.rows = kMaxRowsStep;
  a.qmask = nullptr;
  a.qm_stride = 0;
  a.fxflag = nullptr;
  a.fyflag = nullptr;
  a.fx_stride = 0;
  a.vflag = nullptr;
  a.vf_stride = 0;
  a.skipf = nullptr;
  a.skip_words = 0;
  a.rest = nullptr;
  a.rest_w = a.rest_tiles_x = a.rest_rows = 0;
  a.cfl_tile = nullptr;
  a.cfl_known = 0;
  a.tiles = nullptr;
  a.n_tiles = a.grid_x = a.grid_y = 0;
  a.rest_min = reinterpret_cast<unsigned long long*>(ra + kRaRestMin);
  a.from_rest_min = 0;
  a.dt_from_min = 1;
  const FlagLayout L = flag_layout(a.nx, a.ny, a.pad);
  if (L.fits) {
    unsigned* base = reinterpret_cast<unsigned*>(ra + kRaQFlags);
    a.cfl_tile = reinterpret_cast<unsigned long long*>(base + L.cfl);
    a.qmask = base + L.q;
    a.qm_stride = L.stride;
    a.fyflag = reinterpret_cast<unsigned char*>(base + L.fy);
    a.fxflag = reinterpret_cast<unsigned char*>(base + L.fx);
    a.fx_stride = 4 * L.xtiles;
    a.vflag = reinterpret_cast<unsigned char*>(base + L.v);
    a.vf_stride = 4 * L.vtiles;
    unsigned* marks = base + L.marks;
    a.skipf = reinterpret_cast<unsigned char*>(marks + (tt & 1) * L.sk_words);
    a.skip_words = (int)L.sk_words;
    // The previous step's half, described; take_rest keeps it only when
    // that step was a flagged step on these arrays, and sets its tile height.
    a.rest = reinterpret_cast<unsigned char*>(marks + ((tt + 1) & 1) * L.sk_words);
    const bool prev_x_first = ((tt - 1) % 2 == 0);
    a.rest_w = prev_x_first ? kCols - 1 : kCols;
    a.rest_tiles_x = prev_x_first ? L.xtiles : L.stride;
    a.rest_rows = kMaxRowsStep;
  }
}

}  // namespace

// Mixed form: workspace layout (bytes, each block 256-byte aligned).
namespace {

struct MixedLayout {
  size_t rho_r, e_r, u, v, Qxx, Qyy, F_x, F_y, uF_x, uF_y, vF_x, vF_y, s_r, s_e,
      s_r32, s_e32, total;
};

MixedLayout mixed_layout(int nx, int ny) {
  const size_t nc = (size_t)nx * ny, nf = (size_t)(nx + 1) * (ny + 1);
  MixedLayout L{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) / 256 * 256;
    return at;
  };
  L.rho_r = take(nc * 4);
  L.e_r = take(nc * 4);
  L.u = take(nf * 4);
  L.v = take(nf * 4);
  L.Qxx = take(nc * 4);
  L.Qyy = take(nc * 4);
  L.F_x = take(nf * 4);
  L.F_y = take(nf * 4);
  L.uF_x = take(nf * 4);
  L.uF_y = take(nf * 4);
  L.vF_x = take(nf * 4);
  L.vF_y = take(nf * 4);
  L.s_r = take(nc * 8);
  L.s_e = take(nc * 8);
  L.s_r32 = take(nc * 4);
  L.s_e32 = take(nc * 4);
  L.total = off;
  return L;
}

__global__ void k_make_shadows(size_t n, const double* rho, const double* e,
                               float* rho_r, float* e_r) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    rho_r[i] = f64_to_f32(rho[i]);
    e_r[i] = f64_to_f32(e[i]);
  }
}

}  // namespace

namespace {
// Output rows per CTA of the one-kernel Lagrangian phase.
int g_lag_rows = lagf::kDefaultRows;

// The last flagged step this thread ran, with what identifies its arrays: the
// step after it (and only that one) may take its tile marks (StepArgs::rest)
// and its per-tile CFL minima.
struct RestRecord {
  std::array<const void*, 12> arrays{};
  std::array<const void*, 4> mesh{};     // its spacing arrays
  const void* rho = nullptr;             // the state the step advanced
  const void* e = nullptr;
  const void* ra = nullptr;
  int nx = 0, ny = 0, pad = 0, form = -1, tt = 0;
  StepRows rows;                         // the step's tile heights
  unsigned counts[2 * kListHeights] = {};  // the lengths of the tile lists it left
  bool listed = false;                   // it left tile lists
  bool dense = false;                    // the last lists held nearly every tile
  unsigned long long calls = 0;
  bool valid = false;
  bool follows = false;                  // it directly followed a flagged step
};
thread_local RestRecord t_rest;

constexpr double kDense = 0.8;
constexpr int kDensePeriod = 8;

// Keeps a.rest only when this step directly follows the recorded one on the
// same arrays (and no other mesh call came between), then records this step
// as the one the next may follow (when it runs with flags).  Sets the step's
// tile heights and lists: the previous step's lists unless they hold nearly
// every tile (whose order in the grid is then the better one).
template <typename R>
StepRows take_rest(StepArgs<R>& a, int tt, int form, const std::array<const void*, 12>& arrays,
                   bool flagged, const void* rho, const void* e, double* ra, TileLists& tl,
                   ListArgs& la) {
  const unsigned long long calls = mesh_calls();
  const RestRecord& p = t_rest;
  const std::array<const void*, 4> mesh{a.edgedx, a.edgedy, a.celldx, a.celldy};
  const bool follows = p.valid && flagged && !a.first_step && p.tt + 1 == tt &&
                       p.calls + 1 == calls && p.form == form && p.nx == a.nx &&
                       p.ny == a.ny && p.pad == a.pad && p.arrays == arrays && p.mesh == mesh;
  if (follows) {
    a.rest_rows = p.rows.sweep;
  } else {
    a.rest = nullptr;
  }
  const FlagLayout L = flag_layout(a.nx, a.ny, a.pad);
  unsigned* base = reinterpret_cast<unsigned*>(ra + kRaQFlags);
  // The lists the previous step left, and those this step leaves.
  const size_t list_half = L.list_words[0] + L.list_words[1];
  const unsigned* lists = base + L.lists + ((tt + 1) & 1) * list_half;
  unsigned* out_lists = base + L.lists + (tt & 1) * list_half;
  // (A list entry holds 16 bits for each tile index.)
  const bool listed = flagged && L.list_bands * (kListBand / 2) < 0x10000 && L.list_tx[1] < 0x10000;
  bool use = false, dense = follows && p.dense;
  if (follows && p.listed) {
    const double all = (double)L.list_tx[0] * L.list_bands + (double)L.list_tx[1] * L.list_bands;
    use = p.counts[kListHeights - 1] + p.counts[2 * kListHeights - 1] < kDense * all;
    dense = !use;
  }
  const StepRows rows = pick_step_rows(a.nx, a.ny, a.pad, use ? p.counts : nullptr, flagged,
                                       follows ? &p.rows : nullptr,
                                       Prec<R>::kMixed ? kOverlapMixed : kOverlap64);
  // The per-tile CFL minima are those of tiles of the same height.
  a.cfl_known = follows && p.rows.energy == rows.energy;
  a.rows = rows.lag;
  tl.use = use;
  if (use) {
    a.from_rest_min = a.cfl_known;
    for (int w = 0; w < 2; ++w) {
      for (int h = 0; h < kListHeights; ++h) {
        tl.list[w][h] =
            lists + (w ? L.list_words[0] : 0) + list_offset(L.list_tx[w], L.list_bands, h);
        tl.n[w][h] = (int)p.counts[w * kListHeights + h];
      }
    }
  }
  // Where the last lists held nearly every tile the next are formed eight
  // steps later (10 us a step on a 2048^2 field in motion everywhere).
  const bool build = listed && (!dense || tt % kDensePeriod == 0);
  if (build) {
    const bool x_first = (tt % 2 == 0);
    la.nx = a.nx;
    la.ny = a.ny;
    la.pad = a.pad;
    la.marks = a.skipf;
    la.mark_w = x_first ? kCols - 1 : kCols;
    la.mark_tiles_x = x_first ? L.xtiles : L.stride;
    la.mark_rows = rows.sweep;
    la.bands = L.list_bands;
    const int tx = L.list_tx[0] > L.list_tx[1] ? L.list_tx[0] : L.list_tx[1];
    la.blocks = (int)(((long long)tx * L.list_bands * (kListBand / 2) + kCols - 1) / kCols);
    for (int w = 0; w < 2; ++w) {
      la.tx[w] = L.list_tx[w];
      la.list[w] = out_lists + (w ? L.list_words[0] : 0);
    }
    la.counts = reinterpret_cast<unsigned*>(ra + kRaTileCounts);
    la.cfl_tile = a.cfl_tile;
    la.cfl_tx = L.stride;
    la.cfl_rows = rows.energy;
    la.cfl_ty = (a.ny - 2 * a.pad + rows.energy - 1) / rows.energy;
    la.rest_min = a.rest_min;
  }
  RestRecord r;
  r.arrays = arrays;
  r.mesh = mesh;
  r.rho = rho;
  r.e = e;
  r.ra = ra;
  r.nx = a.nx;
  r.ny = a.ny;
  r.pad = a.pad;
  r.form = form;
  r.tt = tt;
  r.rows = rows;
  r.calls = calls;
  r.valid = flagged;
  r.follows = follows;
  r.listed = build;
  r.dense = dense;
  t_rest = r;
  return rows;
}
}  // namespace

// ---------------------------------------------------------------------------
// Conservation totals by tiles (the reference's print_conservation sums,
// omp3/flow.c:976-994): each tile of interior cells (cons_rows)
// keeps its partial sums (sum rho, sum rho e; each thread down its column, the
// warps and then the four warps of the block in a fixed order) in
// reduce_array, and the last block adds the partials of all tiles in a fixed
// order.  A tile whose cells all lay in tiles the last step's first sweep
// skipped -- at rest through that step, so unchanged since the previous call
// summed them -- keeps its partials without reading a cell.  The totals
// depend only on the cells (the same numbers whichever tiles were kept).
namespace {

struct ConsArgs {
  const double* rho;
  const double* e;
  double* ra;
  double* host;                // page-locked memory for the totals too, or null
  double* part;                // 2 doubles per tile: sum rho, sum rho e
  int nx, ny, pad, tiles_x, tiles, rows;
  const unsigned char* marks;  // the last step's skip marks, or null
  int mark_w, mark_tiles_x, mark_rows;
};

__device__ __forceinline__ double block_sum_fixed(double x, double* s_w) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = x;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < kCols / 32; ++w) t += s_w[w];
  }
  __syncthreads();
  return t;  // (thread 0)
}

__global__ void __launch_bounds__(kCols) k_conservation_tiles(const ConsArgs c) {
  __shared__ double s_w[kCols / 32];
  __shared__ bool s_last;
  const int bx = blockIdx.x % c.tiles_x, by = blockIdx.x / c.tiles_x;
  const int pad = c.pad;
  const int c0 = pad + bx * kConsTile, r0 = pad + by * c.rows;
  const int c1 = min(c0 + kConsTile, c.nx - pad), r1 = min(r0 + c.rows, c.ny - pad);
  bool kept = false;
  if (c.marks) {
    const int b0 = (r0 - pad) / c.mark_rows, b1 = (r1 - 1 - pad) / c.mark_rows;
    const int x0 = (c0 - pad) / c.mark_w, x1 = (c1 - 1 - pad) / c.mark_w;
    const int nxb = x1 - x0 + 1, total = (b1 - b0 + 1) * nxb;
    bool ok = true;
    for (int q = threadIdx.x; q < total; q += blockDim.x) {
      ok = ok && c.marks[(size_t)(b0 + q / nxb) * c.mark_tiles_x + x0 + q % nxb] != 0;
    }
    kept = __syncthreads_and(ok) != 0;
  }
  if (!kept) {
    const int j = c0 + threadIdx.x;
    double ms = 0.0, es = 0.0;
    if (j < c1) {
      // The next eight rows are in flight while these are summed.
      constexpr int kB = 8;
      double rv[kB], ev[kB];
      auto load = [&](int ib) {
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          const bool in = ib + q < r1;  // (rows past the end count as zeros)
          const size_t k = (size_t)(in ? ib + q : r0) * c.nx + j;
          rv[q] = in ? c.rho[k] : 0.0;
          ev[q] = in ? c.e[k] : 0.0;
        }
      };
      load(r0);
      for (int ib = r0; ib < r1; ib += kB) {
        double rc[kB], ec[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          rc[q] = rv[q];
          ec[q] = ev[q];
        }
        if (ib + kB < r1) load(ib + kB);
        ms = __dadd_rn(ms, d_sum8(rc));
#pragma unroll
        for (int q = 0; q < kB; ++q) es = __fma_rn(rc[q], ec[q], es);
      }
    }
    const double tm = block_sum_fixed(ms, s_w);
    const double te = block_sum_fixed(es, s_w);
    if (threadIdx.x == 0) {
      c.part[2 * (size_t)blockIdx.x] = tm;
      c.part[2 * (size_t)blockIdx.x + 1] = te;
    }
  }
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned long long* ticket = reinterpret_cast<unsigned long long*>(c.ra + kRaTicket);
    s_last = (atomicAdd(ticket, 1ull) == (unsigned long long)gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double a = 0.0, b = 0.0;
  // (Eight pairs in flight: one after another the loads took 20 us of a large
  // mesh's call.  The partials are 8-byte aligned, as reduce_array is.)
  constexpr int kP = 8;
  for (int k0 = threadIdx.x; k0 < c.tiles; k0 += kP * kCols) {
    double pm[kP], pe[kP];
#pragma unroll
    for (int q = 0; q < kP; ++q) {
      const int k = k0 + q * kCols;
      pm[q] = k < c.tiles ? __ldcg(c.part + 2 * (size_t)k) : 0.0;
      pe[q] = k < c.tiles ? __ldcg(c.part + 2 * (size_t)k + 1) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kP; ++q) {
      a = __dadd_rn(a, pm[q]);
      b = __dadd_rn(b, pe[q]);
    }
  }
  const double ta = block_sum_fixed(a, s_w);
  const double tb = block_sum_fixed(b, s_w);
  if (threadIdx.x == 0) {
    c.ra[kRaMass] = ta;
    c.ra[kRaEnergy] = tb;
    if (c.host) {
      c.host[0] = ta;
      c.host[1] = tb;
    }
    *reinterpret_cast<unsigned long long*>(c.ra + kRaTicket) = 0ull;
  }
}

// The call the tile partials were last written by, and the mesh-call count
// then: the next call may keep tiles only when exactly one mesh call (the
// step's own) came between.
struct ConsRecord {
  const void* rho = nullptr;
  const void* e = nullptr;
  const void* ra = nullptr;
  int nx = 0, ny = 0, pad = 0;
  unsigned long long calls = 0;
  bool valid = false;
  bool after_step = false;  // right after a flagged step on this state ...
  int step_tt = 0;          // ... of this index
};
thread_local ConsRecord t_cons;

}  // namespace

bool tile_conservation(int nx, int ny, int pad, const double* rho, const double* e,
                       double* ra, double* host, cudaStream_t s) {
  const FlagLayout L = flag_layout(nx, ny, pad);
  if (!L.fits) return false;
  unsigned* base = reinterpret_cast<unsigned*>(ra + kRaQFlags);
  ConsArgs c{};
  c.rho = rho;
  c.e = e;
  c.ra = ra;
  c.host = host;
  c.part = reinterpret_cast<double*>(base + L.cons);
  c.nx = nx;
  c.ny = ny;
  c.pad = pad;
  c.tiles_x = L.cons_tx;
  c.tiles = L.cons_tx * L.cons_ty;
  c.rows = L.cons_h;
  c.marks = nullptr;
  const unsigned long long calls = mesh_calls();
  const RestRecord& p = t_rest;
  const ConsRecord& q = t_cons;
  // Right after a flagged step that advanced this state and directly
  // followed the step after which the partials were last written, on the same
  // arrays, with only that step's own mesh call in between: the state the
  // partials describe is the one that step started from.
  const bool after_step = p.valid && p.calls == calls && p.rho == rho && p.e == e &&
                          p.ra == ra && p.nx == nx && p.ny == ny && p.pad == pad;
  if (after_step && p.follows && q.valid && q.after_step && q.step_tt + 1 == p.tt &&
      q.calls + 1 == calls && q.rho == rho && q.e == e && q.ra == ra && q.nx == nx &&
      q.ny == ny && q.pad == pad) {
    const bool x_first = (p.tt % 2 == 0);
    c.marks = reinterpret_cast<const unsigned char*>(base + L.marks + (p.tt & 1) * L.sk_words);
    c.mark_w = x_first ? kCols - 1 : kCols;
    c.mark_tiles_x = x_first ? L.xtiles : L.stride;
    c.mark_rows = p.rows.sweep;
  }
  // (A fused step leaves the ticket at zero.)
  if (!after_step) cudaMemsetAsync(ra + kRaTicket, 0, sizeof(double), s);
  k_conservation_tiles<<<(unsigned)c.tiles, kCols, 0, s>>>(c);
  count_launches(1);
  ConsRecord r;
  r.rho = rho;
  r.e = e;
  r.ra = ra;
  r.nx = nx;
  r.ny = ny;
  r.pad = pad;
  r.calls = calls;
  r.valid = cudaPeekAtLastError() == cudaSuccess;
  r.after_step = after_step;
  r.step_tt = p.tt;
  t_cons = r;
  return true;
}

int set_lagrangian_rows(int rows) {
  if (rows < 1 || rows > lagf::kMaxRows) {
    return record_error(GB300_ERR_ARG, "gb300_set_lagrangian_rows: %d not in 1 .. %d", rows,
                        lagf::kMaxRows);
  }
  g_lag_rows = rows;
  return GB300_OK;
}

int fused_solve(Mesh* mesh, int tt, double* P, double* rho, double* rho_old,
                double* e, double* u, double* v, double* rho_u, double* rho_v,
                double* Qxx, double* Qyy, double* F_x, double* F_y,
                double* uF_x, double* uF_y, double* vF_x, double* vF_y,
                double* reduce_array, bool one_kernel_lagrangian) {
  if (!reduce_array) return record_error(GB300_ERR_ARG, "solve_hydro_2d: reduce_array is NULL");
  cudaStream_t s = current_stream();
  StepArgs<double> a;
  fill_mesh_args(a, mesh, tt, reduce_array);
  a.rho = rho; a.e = e; a.rho_r = rho; a.e_r = e;
  a.P = P; a.rho_old = rho_old;
  // The Lagrangian phase and the sweeps keep the velocities in uF_y/vF_x (the
  // fused momentum pairs store no fluxes); the advected ones land in u/v.
  a.u = uF_y; a.v = vF_x; a.u_out = u; a.v_out = v;
  a.rho_u = rho_u; a.rho_v = rho_v; a.Qxx = Qxx; a.Qyy = Qyy;
  a.F_x = F_x; a.F_y = F_y; a.uF_x = uF_x; a.uF_y = uF_y; a.vF_x = vF_x;
  a.vF_y = vF_y;
  // The first mass sweep writes into the two cell-sized buffers that hold
  // momentum fluxes later in the step (uF_x, vF_y); the second writes back
  // into rho/e, so neither sweep updates its own input.
  const SweepArgs<double> first{rho, e, rho, e, uF_x, vF_y, uF_x, vF_y};
  const SweepArgs<double> second{uF_x, vF_y, uF_x, vF_y, rho, e, rho, e};
  // The one-kernel Lagrangian phase when asked for and the arrays suit it: it
  // stages rows with 16-byte TMA copies and
  // keeps its change masks in rho_old (the reference's pre-advection density,
  // which the fused sweeps do not read).
  lagf::LagArgs lag{};
  const lagf::LagArgs* lagp = nullptr;
  if (one_kernel_lagrangian) {
    lag.nx = a.nx;
    lag.ny = a.ny;
    lag.pad = a.pad;
    lag.rows = g_lag_rows;
    lag.ntx = (a.nx - 2 * a.pad + 1 + lagf::kW - 1) / lagf::kW;
    const size_t mask_bytes = (size_t)(a.ny + 1) * lag.ntx * lagf::kMaskFields * lagf::kWarps * 4;
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    if (al16(rho) && al16(e) && al16(rho_u) && al16(rho_v) && al16(rho_old) && a.pad == 2 &&
        mask_bytes <= (size_t)a.nx * a.ny * sizeof(double)) {
      lag.edgedx = a.edgedx; lag.edgedy = a.edgedy; lag.celldx = a.celldx; lag.celldy = a.celldy;
      lag.rho = rho; lag.e = e; lag.rho_u = rho_u; lag.rho_v = rho_v;
      lag.u = a.u; lag.v = a.v;
      // Scratch for the changed values: arrays the step writes only later
      // (P is not used by this form; F_x, F_y are the sweeps' outputs).
      lag.e_new = P; lag.rho_u_new = F_x; lag.rho_v_new = F_y;
      lag.masks = reinterpret_cast<unsigned*>(rho_old);
      lag.ra = reduce_array;
      lag.min_slot = a.min_slot;
      lag.mesh = a.mesh;
      lag.dt_slot = a.dt_slot;
      lag.dt = a.dt; lag.dt_h = a.dt_h; lag.max_dt = a.max_dt;
      lag.first_step = a.first_step;
      lagp = &lag;
    }
  }
  TileLists tl;
  ListArgs la{};
  const StepRows sr =
      take_rest(a, tt, 0, {P, rho, e, rho_u, rho_v, uF_y, vF_x, uF_x, vF_y, F_x, F_y, reduce_array},
                a.skipf != nullptr && lagp == nullptr, rho, e, reduce_array, tl, la);
  StepProfiler prof;
  prof.begin(s);
  launch_step(s, a, tt, first, second, prof, sr, tl, la, lagp);
  const int st = finish_step(s, mesh, reduce_array, prof, "solve_hydro_2d (fused)", t_rest.counts);
  if (st != GB300_OK) t_rest.valid = false;
  return st;
}

size_t mixed_workspace_bytes(int nx, int ny) { return mixed_layout(nx, ny).total; }

size_t mixed_zero_block_offset(int nx, int ny) { return mixed_layout(nx, ny).s_r; }

size_t mixed_workspace_offset(int nx, int ny, int field) {
  const MixedLayout L = mixed_layout(nx, ny);
  if (field == GB300_MIXED_U) return L.u;
  if (field == GB300_MIXED_V) return L.v;
  return (size_t)-1;
}

int mixed_prepare(Mesh* mesh, double* rho, double* e, void* work, size_t bytes) {
  const int nx = mesh->local_nx, ny = mesh->local_ny;
  const MixedLayout L = mixed_layout(nx, ny);
  if (!work || bytes < L.total) {
    return record_error(GB300_ERR_ARG,
                        "gb300_mixed_prepare: workspace of %zu bytes, need %zu",
                        bytes, L.total);
  }
  cudaStream_t s = current_stream();
  char* w = static_cast<char*>(work);
  cudaMemsetAsync(work, 0, L.total, s);
  const size_t n = (size_t)nx * ny;
  size_t blocks = (n + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  k_make_shadows<<<(unsigned)blocks, 256, 0, s>>>(
      n, rho, e, reinterpret_cast<float*>(w + L.rho_r),
      reinterpret_cast<float*>(w + L.e_r));
  return check_launch("gb300_mixed_prepare");
}

int mixed_solve(Mesh* mesh, int tt, double* rho, double* e, float* rho_u,
                float* rho_v, void* work, size_t bytes, double* reduce_array) {
  const int nx = mesh->local_nx, ny = mesh->local_ny;
  const MixedLayout L = mixed_layout(nx, ny);
  if (!work || bytes < L.total) {
    return record_error(GB300_ERR_ARG,
                        "gb300_mixed_solve: workspace of %zu bytes, need %zu", bytes,
                        L.total);
  }
  if (!reduce_array) {
    return record_error(GB300_ERR_ARG, "gb300_mixed_solve: reduce_array is NULL");
  }
  char* w = static_cast<char*>(work);
  auto F = [&](size_t off) { return reinterpret_cast<float*>(w + off); };
  auto D = [&](size_t off) { return reinterpret_cast<double*>(w + off); };
  cudaStream_t s = current_stream();
  StepArgs<float> a;
  fill_mesh_args(a, mesh, tt, reduce_array);
  a.rho = rho; a.e = e; a.rho_r = F(L.rho_r); a.e_r = F(L.e_r);
  a.P = nullptr; a.rho_old = nullptr;
  a.u = F(L.uF_y); a.v = F(L.vF_x); a.u_out = F(L.u); a.v_out = F(L.v);
  a.rho_u = rho_u; a.rho_v = rho_v;
  a.Qxx = F(L.Qxx); a.Qyy = F(L.Qyy); a.F_x = F(L.F_x); a.F_y = F(L.F_y);
  a.uF_x = F(L.uF_x); a.uF_y = F(L.uF_y); a.vF_x = F(L.vF_x); a.vF_y = F(L.vF_y);
  const SweepArgs<float> first{rho, e, a.rho_r, a.e_r, D(L.s_r), D(L.s_e),
                               F(L.s_r32), F(L.s_e32)};
  const SweepArgs<float> second{D(L.s_r), D(L.s_e), F(L.s_r32), F(L.s_e32),
                                rho, e, a.rho_r, a.e_r};
  TileLists tl;
  ListArgs la{};
  const StepRows sr =
      take_rest(a, tt, 1, {rho, e, rho_u, rho_v, work, reduce_array, nullptr, nullptr, nullptr,
                           nullptr, nullptr, nullptr},
                a.skipf != nullptr, rho, e, reduce_array, tl, la);
  StepProfiler prof;
  prof.begin(s);
  launch_step(s, a, tt, first, second, prof, sr, tl, la);
  const int st = finish_step(s, mesh, reduce_array, prof, "gb300_mixed_solve", t_rest.counts);
  if (st != GB300_OK) t_rest.valid = false;
  return st;
}

}  // namespace flow
