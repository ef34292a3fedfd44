// GLST device kernels for sm_100a (B200).
//
// Data layout in HBM (one system):
//   pk[N]      float4 (dx, dy, dz, q): cell-ordered atoms, position relative
//              to the centre of the atom's cell, computed in FP64 and rounded
//   pd[N]      double4 (x, y, z, q): cell-ordered atoms, FP64 absolute
//   S[C][K]    float2: cell-relative structure factor sum_j q_j e^{-ik.(r_j - c)}
//              of every cell at every node (FP32 per atom tile, FP64 across
//              tiles, stored rounded to FP32)
//   R[C][K]    float2: shell sum times weight times e^{+ik.c} (cell centre c)
//   part[P][N] double4: long-range partial sums, one row per node chunk
//   sr[W][N]   double4: near-field sums, one row per row of neighbour cells
// Cell c = (ix*ny + iy)*nz + iz, as in the reference (src/glst_force.cu:379-382).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace glst {
namespace dev {

struct Grid {
  uint32_t nx, ny, nz, ncell;
  double l;       // cell edge (CT value widened to double)
  int ct_float;   // bin in float arithmetic (glst_force<float>)
};

// Layout of the structure factors S and shell sums R (C cells x K nodes):
// blocks of kNodeBlock consecutive nodes, each block cell-major, so that a
// cell's run of nodes is contiguous within a block (the structure-factor
// stores and the long-range loads) and one node's values over all cells lie
// in one C x kNodeBlock region (the shell-sum loads and stores; a plain
// cell-major layout put them a whole row apart, one page per cell).
// Buffers hold C x ceil(K / kNodeBlock) x kNodeBlock elements.
constexpr uint32_t kNodeBlock = 32;
__host__ __device__ __forceinline__ size_t sr_index(uint32_t c, uint32_t k, uint32_t ncell) {
  return ((size_t)(k / kNodeBlock) * ncell + c) * kNodeBlock + (k % kNodeBlock);
}

__device__ __forceinline__ double cell_centre(uint32_t i, double l) {
  return (static_cast<double>(i) + 0.5) * l;
}

// Arguments of the shell sums (shell_sums.cuh).
struct SatArgs {
  const float2 *S;               // cell-relative structure factors
  const double4 *node64;        // (kx, ky, kz, w) FP64
  const uint32_t *node_radii;   // r_in | r_out << 16
  uint32_t K;                   // nodes handled by this launch
  uint32_t kbase;               // local index of the launch's first node in S and R
  uint32_t nb;                  // nodes per CTA (a power of two, <= 32)
  uint32_t lg_nb;               // log2(nb)
  uint32_t xyz_table;           // 1: cell coordinates tabulated in shared memory
  uint32_t stride;              // shared row stride (complex), >= ncell, = 1 (mod 8)
  float2 *R;
};

}  // namespace dev
}  // namespace glst
