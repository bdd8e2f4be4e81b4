// common.cuh -- shared definitions of the GB300 flow kernel set.
//
// Grid conventions follow the reference kernel set (omp3/flow.c): nx, ny are
// the padded cell counts (local_nx/local_ny), pad = 2 ghost layers.
//   cell   (ii,jj): ii*nx + jj           ny rows,     nx cols
//   x-face (ii,jj): ii*(nx+1) + jj       ny rows,     nx+1 cols
//   y-face (ii,jj): ii*nx + jj           ny+1 rows,   nx cols (omp3/flow.c:129)
//   corner (ii,jj): ii*(nx+1) + jj       ny+1 rows,   nx+1 cols
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace flow {

// Physical constants of flow_interface.h:7-9 and flow_data.h:5.
constexpr double kGam = 1.4;
constexpr double kCQ = 3.0;
constexpr double kCT = 0.3;
#define FLOW_C_M (1.5 / 0.3)

// Layout of the caller's reduce_array (flow_interface.h:20).  The host driver
// allocates it with local_nx*local_ny doubles (arch SharedData), and the
// kernel set uses it as its only device scratch:
//   [0] dt, [1] dt_h          device copy of the timestep pair
//   [2] ticket                block-completion counter (uint64 bits)
//   [3] mass, [4] energy      conservation totals of the last reduction
//   [5] status                error word of the fused kernels (uint64 bits)
//   [6] CFL minimum           running minimum of the fused step's CFL
//                             candidates (uint64 bits of a non-negative
//                             double: bit order = value order)
//   [7] mesh                  eight bytes, one of each part of the mesh test:
//                             bit 0 uniform, bit 1 spacings all powers of two,
//                             bits 2 and 3 some of them (StepArgs::mesh),
//                             formed on the device at the start of a step,
//                             with the
//   [8 .. 11] spacings        dx, dy, 1/dx, 1/dy of a uniform mesh
//   [12] minimum at rest      the CFL minimum over the shock-heating tiles
//                             the next step need not visit (as [6])
//   [13 .. 16] tile counts    lengths of the next step's tile lists (uint32,
//                             128- and 127-column tiles of 2, 4, 8, 16 rows)
//   [17 ...]                  per-block partials (2 doubles per block, at
//                             most kMaxReduceBlocks blocks)
//   [kRaQFlags ...]           the fused step's tile flags, when the array
//                             is large enough to hold them: per-tile CFL
//                             minima, then the viscous-stress, mass-flux and
//                             velocity flags, the two halves of the sweeps'
//                             skip marks and the tile lists (fused.cu,
//                             fill_mesh_args)
enum : int {
  kRaDt = 0,
  kRaDtH = 1,
  kRaTicket = 2,
  kRaMass = 3,
  kRaEnergy = 4,
  kRaStatus = 5,
  kRaMinBits = 6,
  kRaMesh = 7,
  kRaRestMin = 12,
  kRaTileCounts = 13,
  kRaPartial = 17,
};
constexpr int kMaxReduceBlocks = 1024;
constexpr int kRaQFlags = kRaPartial + 2 * kMaxReduceBlocks;

// Ghost-fill modes of handle_boundary_2d (arch; omp3/flow.c:156).
enum : int { kNoInvert = 0, kInvertX = 1, kInvertY = 2 };

// Indices are never negative here, so they are formed with one 32x32->64-bit
// unsigned multiply-add (a signed int widened to size_t first costs a 64-bit
// multiply).
__host__ __device__ inline size_t cidx(int nx, int ii, int jj) {
  return (size_t)(unsigned)ii * (unsigned)nx + (unsigned)jj;
}
__host__ __device__ inline size_t fidx(int nx, int ii, int jj) {
  return (size_t)(unsigned)ii * (unsigned)(nx + 1) + (unsigned)jj;
}

// Ordinary minimum (first argument when strictly smaller).
__device__ __forceinline__ double dmin(double a, double b) {
  return (a < b) ? a : b;
}

}  // namespace flow
