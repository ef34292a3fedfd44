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

// ----------------------------------------------------------------------------
// How the work over cells is divided (host and device).
constexpr uint32_t kSms = 148;        // B200
constexpr uint32_t kSortCells = 8;    // cells per CTA, sparse grids

// Cells per CTA of the sort.
__host__ __device__ inline uint32_t sort_cells(uint32_t natom, uint32_t ncell) {
  return natom / ncell <= 16 ? kSortCells : 1u;
}

// Cells per structure-factor CTA, for `quads` quads of direction tiles.  The
// group's table is copied once per CTA, so more cells help where they hold few
// atoms and CTAs are still many: eight from 28 CTAs per SM on, four from 24
// (12 at eight cells each).  Measured, one / four / eight cells, us: 26^3 cells
// of 5 atoms at 1e-3 320 / 241 / 231 (11,000 CTAs of eight cells); 16^3 70 / 60
// / 64 (2,000); 8^3 at the default order 222 / 223 / 239 (1,900); 6^3 93 / 100 /
// 117 (700); 3^3 20 / 32 / 55 (50).  (A batch's systems count the quads of all
// that run beside each other: 24 boxes of 8^3 cells at 1e-4, 4.8 ms a pass
// against 4.9 with one cell per CTA.)
__host__ __device__ inline uint32_t sf_cells(uint32_t natom, uint32_t ncell, uint32_t quads) {
  const uint64_t ctas = (uint64_t)ncell * quads / 8;
  return natom / ncell > 16 || ctas < 12 * kSms ? 1u : ctas < 28 * kSms ? 4u : 8u;
}

// Atoms of a cell that the cell's own warps of the near field and the gather
// take, at most: 2.5 times the mean, in whole 32s.  Evenly filled boxes stay
// below it (from 4 cells per axis on their full cells hold at most 2.4 times the
// mean of a grid whose outer layers are empty); at 1.25 times the mean full
// cells were cut just before their end, which cost batches of such boxes 2.5 %.
// The rest of a denser cell (a droplet or a slab in a wide box: the mean says
// nothing about its cells) is listed by the scan as pieces of up to kPieceAtoms
// atoms, and the last kPieceWarps warps of a near-field row or a gather chunk take
// pieces when they are done with their own cell (the outer layers are the emptiest;
// on large grids the others' look at the list would cost 0.7 %).
// Measured, all of a cell's atoms by its own warps against this: near field of
// 8,000 atoms in one of 26^3 cells 167 against 0.9 ms, 12,000 atoms in a droplet
// on 20^3 cells 1.6 against 0.21 ms and their gather 0.46 against 0.14.
constexpr uint32_t kPieceAtoms = 32;
constexpr uint32_t kPieceWarps = 2048;
__host__ __device__ inline uint32_t cell_cap(uint32_t natom, uint32_t ncell) {
  const uint64_t cap = ((uint64_t)natom * 5 / 2 / ncell + kPieceAtoms) / kPieceAtoms * kPieceAtoms;
  return cap < natom ? (uint32_t)cap : (natom + kPieceAtoms) / kPieceAtoms * kPieceAtoms;
}

// Pieces there can be: every piece's cell holds another 32 atoms of its own.
__host__ __device__ inline uint32_t max_pieces(uint32_t natom, uint32_t ncell) {
  return natom > cell_cap(natom, ncell) ? natom / kPieceAtoms : 0u;
}

// The list of pieces: {cell, first atom within the cell}.
struct Pieces {
  const uint2 *list;
  const uint32_t *n;
  uint32_t cap;  // cell_cap
};

// Lanes per chunk, at most: the widest chunks of which there are still 2,048
// (about four warps for each of the GPU's schedulers), else 8 atoms wide.
__host__ __device__ inline uint32_t sr_width(uint32_t natom, uint32_t rows) {
  const uint64_t lanes = (uint64_t)natom * rows;
  return lanes >= 2048u * 32u ? 32u : lanes >= 2048u * 16u ? 16u : 8u;
}

// Near-field CTAs per SM: four (128 registers) where warps have many atoms to
// pair, five where cells hold few and latency counts.  Measured, four against
// five: 87 atoms per cell 157 against 167 us, 168 per cell 175 against 192, 6 per
// cell on 26^3 cells 105 against 98.
__host__ __device__ inline int sr_ctas(uint32_t natom, uint32_t ncell) { return natom / ncell > 16 ? 4 : 5; }

// Near-field CTAs (four warps) for the cells of one row.
__host__ __device__ inline uint32_t sr_blocks(uint32_t ncell, uint32_t warps_per_cell) {
  return (uint32_t)(((uint64_t)ncell * warps_per_cell + 3) / 4);
}

// Warps per cell for a mean number of atoms per cell.
__host__ __device__ inline uint32_t sr_warps_per_cell(uint32_t natom, uint32_t ncell, uint32_t width) {
  const uint32_t mean = natom / ncell;
  return 4 * mean <= 3 * width ? 1u : 4 * mean <= 7 * width ? 2u : 4u;
}

}  // namespace dev
}  // namespace glst
