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

constexpr unsigned kSortCap = 8192;   // atoms per cell the shared-memory cell sort holds

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

// SFU sine and cosine of an FP32 angle in radians (PTX sin/cos.approx,
// flush-to-zero).  Absolute error ~1e-6 for the |x| < ~30 rad used here,
// below the FP32 rounding of the phase itself at that magnitude.
__device__ __forceinline__ void sfu_sincos(float x, float *s, float *c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}

__device__ __forceinline__ double cell_centre(uint32_t i, double l) {
  return (static_cast<double>(i) + 0.5) * l;
}

// ----------------------------------------------------------------------------
// Cell assignment.  Binning follows calc_cell_atom_count_kernel
// (src/glst_force.cu:356-386): the coordinate (converted to CT) times 1/l in
// CT, truncated toward zero, clamped to [0, n-1].
__device__ __forceinline__ uint32_t bin_axis(double r, const Grid &g, uint32_t n) {
  int c;
  if (g.ct_float) {
    const float inv = __fdiv_rn(1.0f, static_cast<float>(g.l));
    c = static_cast<int>(__fmul_rn(static_cast<float>(r), inv));
  } else {
    const double inv = __ddiv_rn(1.0, g.l);
    c = static_cast<int>(__dmul_rn(r, inv));
  }
  c = (c >= static_cast<int>(n)) ? static_cast<int>(n) - 1 : c;
  c = (c < 0) ? 0 : c;
  return static_cast<uint32_t>(c);
}

// K_bin: cell of every atom and an (unordered) slot inside the cell.
// (Each kernel's body is a device function of its block indices, so that
// the batched work-list kernels can run the same code for many systems.)
__device__ __forceinline__ void bin_block(const double *__restrict__ rx, const double *__restrict__ ry,
                                          const double *__restrict__ rz, uint32_t n, const Grid &g,
                                          uint32_t *__restrict__ atom_cell, uint32_t *__restrict__ atom_slot,
                                          uint32_t *__restrict__ cell_count, uint32_t bx) {
  const uint32_t i = bx * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t cx = bin_axis(rx[i], g, g.nx);
  const uint32_t cy = bin_axis(ry[i], g, g.ny);
  const uint32_t cz = bin_axis(rz[i], g, g.nz);
  const uint32_t cell = (cx * g.ny + cy) * g.nz + cz;
  atom_cell[i] = cell;
  atom_slot[i] = atomicAdd(&cell_count[cell], 1u);
}

__global__ void k_bin(const double *__restrict__ rx, const double *__restrict__ ry,
                      const double *__restrict__ rz, uint32_t n, Grid g,
                      uint32_t *__restrict__ atom_cell, uint32_t *__restrict__ atom_slot,
                      uint32_t *__restrict__ cell_count) {
  bin_block(rx, ry, rz, n, g, atom_cell, atom_slot, cell_count, blockIdx.x);
}

// K_scan: exclusive offsets of the cell counts (one CTA of 1024 threads, four
// consecutive cells per thread and step: 26^3 cells in 5 steps instead of 18).
__device__ __forceinline__ void scan_body(const uint32_t *__restrict__ cell_count, uint32_t ncell,
                                          uint32_t *__restrict__ cell_point) {
  __shared__ uint32_t warp_sums[32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < ncell; base += 4 * blockDim.x) {
    const uint32_t c = base + 4 * threadIdx.x;
    uint32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = (c + u < ncell) ? cell_count[c + u] : 0u;
    const uint32_t mine = v[0] + v[1] + v[2] + v[3];
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (unsigned)o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t s = (lane < nw) ? warp_sums[lane] : 0u;  // every warp scans the warps' sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= (unsigned)o) s += y;
    }
    const uint32_t before_warp = __shfl_sync(0xffffffffu, s, (warp + 31) & 31u);
    uint32_t p = carry + (warp ? before_warp : 0u) + (x - mine);
    carry += __shfl_sync(0xffffffffu, s, 31);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (c + u < ncell) cell_point[c + u] = p;
      p += v[u];
    }
    __syncthreads();  // warp_sums is rewritten
  }
}

__global__ void k_scan(const uint32_t *__restrict__ cell_count, uint32_t ncell,
                       uint32_t *__restrict__ cell_point) {
  scan_body(cell_count, ncell, cell_point);
}

__device__ __forceinline__ void scatter_block(const uint32_t *__restrict__ atom_cell,
                                              const uint32_t *__restrict__ atom_slot,
                                              const uint32_t *__restrict__ cell_point, uint32_t n,
                                              uint32_t *__restrict__ perm, uint32_t bx) {
  const uint32_t i = bx * blockDim.x + threadIdx.x;
  if (i >= n) return;
  perm[cell_point[atom_cell[i]] + atom_slot[i]] = i;
}

__global__ void k_scatter(const uint32_t *__restrict__ atom_cell,
                          const uint32_t *__restrict__ atom_slot,
                          const uint32_t *__restrict__ cell_point, uint32_t n,
                          uint32_t *__restrict__ perm) {
  scatter_block(atom_cell, atom_slot, cell_point, n, perm, blockIdx.x);
}

// K_sort_pack.  The atomics of k_bin leave the atoms of a cell in arbitrary
// order; sorting each cell's indices ascending reproduces the order of a
// stable sort by cell id (the reference's CUB radix sort,
// src/glst_force.cu:510-517).  Then writes the packets.  A CTA takes one cell
// (bitonic sort), or on sparse grids kSortCells cells: one warp each for cells
// of up to kSortWarpCap atoms, an atom's place being the number of smaller
// indices, then the whole CTA for each larger one.  Launched with 32
// kSortCells threads and kSortCap u32 of dynamic shared memory.
constexpr uint32_t kSortCells = 8;
constexpr uint32_t kSortWarpCap = 32;
__host__ __device__ inline uint32_t sort_cells(uint32_t natom, uint32_t ncell) {  // cells per CTA
  return natom / ncell <= 16 ? kSortCells : 1u;
}
__device__ __forceinline__ void pack_atom(uint32_t slot, uint32_t a, double cx, double cy, double cz,
                                          const double *__restrict__ rx, const double *__restrict__ ry,
                                          const double *__restrict__ rz, const double *__restrict__ qc,
                                          uint32_t *__restrict__ sorted_idx, float4 *__restrict__ pk,
                                          double4 *__restrict__ pd) {
  const double x = rx[a], y = ry[a], z = rz[a], q = qc[a];
  sorted_idx[slot] = a;
  pd[slot] = make_double4(x, y, z, q);
  pk[slot] = make_float4(static_cast<float>(x - cx), static_cast<float>(y - cy), static_cast<float>(z - cz),
                         static_cast<float>(q));
}

__device__ __forceinline__ void sort_pack_block(const uint32_t *__restrict__ perm,
                                                const uint32_t *__restrict__ cell_count,
                                                const uint32_t *__restrict__ cell_point, const Grid &g,
                                                const uint32_t *__restrict__ atom_cell, uint32_t natom,
                                                const double *__restrict__ rx, const double *__restrict__ ry,
                                                const double *__restrict__ rz, const double *__restrict__ qc,
                                                uint32_t *__restrict__ sorted_idx, float4 *__restrict__ pk,
                                                double4 *__restrict__ pd, uint32_t cell) {
  extern __shared__ uint32_t s_idx[];  // the whole CTA's
  const uint32_t cnt = cell_count[cell];
  const uint32_t start = cell_point[cell];
  if (cnt == 0) return;
  const uint32_t ix = cell / (g.ny * g.nz), iy = (cell / g.nz) % g.ny, iz = cell % g.nz;
  const double cx = cell_centre(ix, g.l), cy = cell_centre(iy, g.l), cz = cell_centre(iz, g.l);
  if (cnt > kSortCap) {
    // Too many atoms for the shared-memory sort: an atom's place in the cell
    // is the number of atoms of the cell with a smaller index, found by one
    // pass over every atom's cell in index order (per step: a warp ballot per
    // warp, then the counts of the warps before).  Stable by construction;
    // O(natom) per such cell, which only dense grids have.
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t seen = 0;
    for (uint32_t i0 = 0; i0 < natom; i0 += blockDim.x) {
      const uint32_t i = i0 + threadIdx.x;
      const bool mine = i < natom && atom_cell[i] == cell;
      const uint32_t bal = __ballot_sync(0xffffffffu, mine);
      if (lane == 0) s_idx[warp] = __popc(bal);
      __syncthreads();
      uint32_t before = seen, total = seen;
      for (uint32_t w = 0; w < nw; w++) {
        const uint32_t c = s_idx[w];
        before += (w < warp) ? c : 0u;
        total += c;
      }
      if (mine) sorted_idx[start + before + __popc(bal & ((1u << lane) - 1u))] = i;
      seen = total;
      __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x)
      pack_atom(start + i, sorted_idx[start + i], cx, cy, cz, rx, ry, rz, qc, sorted_idx, pk, pd);
    return;
  }
  uint32_t np2 = 1;
  while (np2 < cnt) np2 <<= 1;
  for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x)
    s_idx[i] = (i < cnt) ? perm[start + i] : 0xffffffffu;
  __syncthreads();
  // bitonic sort, ascending
  for (uint32_t k = 2; k <= np2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < np2; i += blockDim.x) {
        const uint32_t p = i ^ j;
        if (p > i) {
          const uint32_t a = s_idx[i], b = s_idx[p];
          const bool up = ((i & k) == 0);
          if ((a > b) == up) {
            s_idx[i] = b;
            s_idx[p] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x)
    pack_atom(start + i, s_idx[i], cx, cy, cz, rx, ry, rz, qc, sorted_idx, pk, pd);
}

__device__ __forceinline__ void sort_pack_cells(const uint32_t *__restrict__ perm,
                                                const uint32_t *__restrict__ cell_count,
                                                const uint32_t *__restrict__ cell_point, const Grid &g,
                                                const uint32_t *__restrict__ atom_cell, uint32_t natom,
                                                const double *__restrict__ rx, const double *__restrict__ ry,
                                                const double *__restrict__ rz, const double *__restrict__ qc,
                                                uint32_t *__restrict__ sorted_idx, float4 *__restrict__ pk,
                                                double4 *__restrict__ pd, uint32_t bx) {
  extern __shared__ uint32_t s_idx[];
  if (sort_cells(natom, g.ncell) == 1) {
    sort_pack_block(perm, cell_count, cell_point, g, atom_cell, natom, rx, ry, rz, qc, sorted_idx, pk, pd, bx);
    return;
  }
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t cell = bx * kSortCells + warp;
  const uint32_t cnt = cell < g.ncell ? cell_count[cell] : 0u;
  if (cnt > 0 && cnt <= kSortWarpCap) {
    const uint32_t start = cell_point[cell];
    uint32_t *mine = s_idx + warp * kSortWarpCap;
    for (uint32_t i = lane; i < cnt; i += 32) mine[i] = perm[start + i];
    __syncwarp();
    const uint32_t ix = cell / (g.ny * g.nz), iy = (cell / g.nz) % g.ny, iz = cell % g.nz;
    const double cx = cell_centre(ix, g.l), cy = cell_centre(iy, g.l), cz = cell_centre(iz, g.l);
    for (uint32_t i = lane; i < cnt; i += 32) {
      const uint32_t a = mine[i];
      uint32_t rank = 0;
#pragma unroll 8
      for (uint32_t j = 0; j < cnt; j++) rank += mine[j] < a ? 1u : 0u;
      pack_atom(start + rank, a, cx, cy, cz, rx, ry, rz, qc, sorted_idx, pk, pd);
    }
  }
  if (!__syncthreads_or(cnt > kSortWarpCap)) return;
  for (uint32_t w = 0; w < kSortCells; w++) {
    const uint32_t c = bx * kSortCells + w;
    if (c < g.ncell && cell_count[c] > kSortWarpCap) {
      sort_pack_block(perm, cell_count, cell_point, g, atom_cell, natom, rx, ry, rz, qc, sorted_idx, pk, pd, c);
      __syncthreads();
    }
  }
}

__global__ void k_sort_pack(const uint32_t *__restrict__ perm,
                            const uint32_t *__restrict__ cell_count,
                            const uint32_t *__restrict__ cell_point, Grid g,
                            const uint32_t *__restrict__ atom_cell, uint32_t natom,
                            const double *__restrict__ rx, const double *__restrict__ ry,
                            const double *__restrict__ rz, const double *__restrict__ qc,
                            uint32_t *__restrict__ sorted_idx, float4 *__restrict__ pk,
                            double4 *__restrict__ pd) {
  sort_pack_cells(perm, cell_count, cell_point, g, atom_cell, natom, rx, ry, rz, qc, sorted_idx, pk, pd,
                  blockIdx.x);
}

// ----------------------------------------------------------------------------
// Sine and cosine on the FP32 FMA pipe, for part of the (atom, node) pairs so
// that the FMA pipe carries some of the work the MUFU pipe would otherwise
// serialise.  Method: theta = n pi + r with n = rint(theta / pi) (rounded by
// adding 1.5 * 2^23), r = theta - n pi in two FMA steps (pi = kPiHi + kPiLo,
// kPiHi with 8 significant bits so n * kPiHi is exact), then
//   sin r = r + r^3 P(r^2),  cos r = Q(r^2)   on |r| <= pi/2,
// with P of degree 3 and Q of degree 4, coefficients fitted by this project
// (Lawson-weighted least squares on [0, (pi/2)^2], csrc/fit_sincos.py).
// sin(theta) = (-1)^n sin r, cos(theta) = (-1)^n cos r: the common sign is
// returned folded into a factor (the atom's charge) instead of applied to
// both results.  Max abs error 1.8e-7 for |theta| <= 30.
constexpr float kInvPi = 0.318309886183790672f;
constexpr float kRoundMagic = 12582912.0f;  // 1.5 * 2^23
constexpr float kPiHi = 3.140625f;
constexpr float kPiLo = 9.67653589793e-4f;
constexpr float kSin1 = -0.16666658222675323f, kSin2 = 0.008333051577210426f,
                kSin3 = -0.000198090827325359f, kSin4 = 2.6052375687868334e-06f;
constexpr float kCos0 = 0.9999999403953552f, kCos1 = -0.4999990463256836f, kCos2 = 0.04166358709335327f,
                kCos3 = -0.0013853712007403374f, kCos4 = 2.3154068912845105e-05f;

__device__ __forceinline__ void fma_sincos_signed(float th, float q, float *s, float *c, float *qs) {
  const float t = fmaf(th, kInvPi, kRoundMagic);
  const float n = t - kRoundMagic;
  float r = fmaf(-n, kPiHi, th);
  r = fmaf(-n, kPiLo, r);
  const float r2 = r * r;
  float p = fmaf(kSin4, r2, kSin3);
  p = fmaf(p, r2, kSin2);
  p = fmaf(p, r2, kSin1);
  *s = fmaf(p * r2, r, r);
  float cc = fmaf(kCos4, r2, kCos3);
  cc = fmaf(cc, r2, kCos2);
  cc = fmaf(cc, r2, kCos1);
  *c = fmaf(cc, r2, kCos0);
  *qs = __int_as_float(__float_as_int(q) ^ (__float_as_int(t) << 31));
}

// Operand pairs of the paired FP32 instructions (FFMA2/FADD2: two IEEE FP32
// operations per instruction).
__device__ __forceinline__ float2 bcast(float v) { return make_float2(v, v); }

// ----------------------------------------------------------------------------
// Structure factors.  S_c(k) = sum_{j in c} q_j e^{-i k.r_j}
//                            = e^{-i k.c} sum_j q_j e^{-i k.d_j},  d_j = r_j - c.
// Nodes are k = kappa_r s (group -> direction -> radial).  On a direction's
// ray every phase is kappa_r u with one u = s.d_j, |u| <= U (U: the cell's
// circumscribed sphere and a margin), and
//   e^{-i kappa u} = sum_p (2 - [p = 0]) (-i)^p J_p(kappa U) T_p(u / U)
// (Jacobi-Anger) falls off faster than geometrically beyond p = kappa U (18,
// 8 and 4 rad in water10k's groups): P = 36, 24 and 16 terms carry all 33,
// 27 and 19 radial nodes to below the rounding of an FP32 phase.  So a
// direction takes P real moments sum_j q_j T_p(x_j), one FMA each per atom,
// and one P x n_rad product per cell -- where one sine and cosine per (atom,
// node) kept the SFU and FMA pipes full (water10k 1.11 ms).
//
// The moments are formed in the product basis T_{Bg} T_b (b < B, p = Bg + b):
// B + P/B recurrence steps and P accumulations per atom instead of P and P.
// The host expands the Jacobi-Anger series in that basis in FP64
// (cheb_product_basis); B is even, so even b feed the real part of S and odd
// b the imaginary part, and a pair (b, b + 1) is one FFMA2 both when it is
// accumulated and when it is multiplied out.
//
// A CTA's four warps take 32 directions of one group each, lane = direction,
// moments in registers, atoms broadcast from shared memory, for one cell
// (sparse grids: eight); the group's table is copied to shared memory once (read through L1
// as broadcasts it took five wavefronts per 16 bytes, and half of L1's time).
// After that the warps are independent.  FP32 over a tile of <=
// kSfAtomTile atoms, then FP64 over the tiles of a denser cell.  S is stored
// cell-relative in FP32; its twiddle e^{-ik.c} is applied by the shell sums
// as they load S.  Atoms beyond U (outside the box by more than the margin,
// or not a number) and tiles of too few atoms for the product (16 atoms cost
// as much as P terms) take one sine and cosine per node instead.
// Measured: water10k 1.112 -> 0.297 ms, 1,000 waters on 4^3 cells 0.144 ->
// 0.056 ms, 168 atoms per cell 0.313 -> 0.094 ms; forces 3.3e-8 -> 1.5e-8 off
// the FP64 path.
constexpr int kSfWarps = 4;
constexpr int kSfThreads = 32 * kSfWarps;
constexpr int kSfAtomTile = 128;
constexpr int kSfRadChunk = 64;   // radial nodes staged at a time, at most
constexpr int kChebMaxP = 64;     // series terms, at most (even to 48, then multiples of 4)
__host__ __device__ constexpr int cheb_b(int P) { return P > 24 ? 8 : 4; }
__host__ __device__ constexpr int cheb_row(int P) { return (P + 3) / 4 * 4; }  // table row, in floats

// Up to 32 directions of one group (none: padding, so that a group's tiles are
// whole quads).
struct DirTile {
  uint32_t node_begin;   // local internal index of (first direction, r = 0)
  uint32_t dir_begin;    // global direction index of the first direction
  uint32_t n_dir;        // directions in the tile (<= 32)
  uint32_t n_rad;        // radial nodes per direction in this group
  uint32_t P;            // series terms, even (0: one sincos per node)
  uint32_t tab;          // offset of the group's n_rad x cheb_row(P) table
  uint32_t kappa_begin;  // offset of this group's radial table
  uint32_t lr_P, lr_tab; // the gather's series terms and table
};

// Per-handle constants of the series: 1 / U and the largest |d|^2 it takes.
struct ChebScale {
  float inv_u, u2;
};

// Arguments of the structure factors.  Tiles index nodes by the handle's
// local node; S holds the nodes from node_off on (a node range of the handle:
// the whole of it, or one stage).
struct SfArgs {
  const float4 *pk;
  const uint32_t *cell_count, *cell_point;
  const DirTile *tiles;
  const float4 *dirs;
  const float *kappa;
  const float4 *tab;   // product-basis series, cheb_row(P) floats per radial node
  float2 *S, *lo_buf;  // lo_buf: scratch of S's size
  ChebScale cs;
  uint32_t ncell, n_tiles, max_rad, node_off;
  uint32_t tab4;       // float4s of the largest group's table
  uint32_t cells;      // cells per CTA
};

// Cells per structure-factor CTA: one (four cost 5 % on water10k, 40 % on 1,000
// waters), but eight where a cell's few atoms take less than copying the table
// (26^3 cells of 6 atoms: 0.32 ms with one, 0.24 with four).
__host__ __device__ inline uint32_t sf_cells(uint32_t natom, uint32_t ncell) { return natom / ncell <= 16 ? 8u : 1u; }

// Rows of the staged results are an odd number of float2 apart (bank spread).
__host__ __device__ constexpr uint32_t sf_row(uint32_t rc) { return rc | 1u; }

__host__ __device__ inline size_t sf_smem_bytes(uint32_t max_rad, uint32_t tab4) {
  const uint32_t rc = max_rad < (uint32_t)kSfRadChunk ? max_rad : (uint32_t)kSfRadChunk;
  return tab4 * sizeof(float4) + (size_t)kSfWarps * (32 * sizeof(float4) + 32 * sf_row(rc) * sizeof(float2));
}

// The general form, one sine and cosine per (atom, node), added to the staged
// results: the tile's atoms beyond the series' range (all: every atom).
__device__ __noinline__ void sf_direct(const float4 *__restrict__ pk, uint32_t na, bool all, float u2, float4 s,
                                       const float *__restrict__ kappa, uint32_t rc, float2 *__restrict__ row) {
  for (uint32_t r = 0; r < rc; r++) {
    const float kap = kappa[r];
    float fr = 0.f, fi = 0.f;
    for (uint32_t j = 0; j < na; j++) {
      const float4 p = pk[j];
      if (!all && fmaf(p.x, p.x, fmaf(p.y, p.y, p.z * p.z)) <= u2) continue;
      const float u = fmaf(s.x, p.x, fmaf(s.y, p.y, s.z * p.z));
      float sn, cs, qs;
      fma_sincos_signed(kap * u, p.w, &sn, &cs, &qs);
      fr = fmaf(qs, cs, fr);
      fi = fmaf(qs, sn, fi);
    }
    const float2 o = row[r];
    row[r] = make_float2(o.x + fr, o.y - fi);
  }
}

// A cell of several tiles adds them in FP64: the running sum is kept between
// tiles as an unevaluated pair of floats, the leading part in S and the
// remainder in lo_buf (the shell sums' output buffer, which is free until
// the structure factors are done); the last tile stores the sum rounded once
// to FP32.  Out of line, so that the registers of this rare path do not
// count against the hot loop's.
__device__ __noinline__ void sf_store_dense(float2 f, size_t o, bool add, bool last, float2 *__restrict__ S,
                                            float2 *__restrict__ lo_buf) {
  double vx = f.x, vy = f.y;
  if (add) {
    const float2 h = S[o], l = lo_buf[o];
    vx += (double)h.x + (double)l.x;
    vy += (double)h.y + (double)l.y;
  }
  const float hx = static_cast<float>(vx), hy = static_cast<float>(vy);
  S[o] = make_float2(hx, hy);
  if (!last) lo_buf[o] = make_float2(static_cast<float>(vx - hx), static_cast<float>(vy - hy));
}

// Moments of one tile of atoms in N (pairs (b, b + 1) of the product basis).
// The zeroth, the tile's charge, is the same for every direction and node, so
// the rounding of an FP32 sum would act as a point charge at the cell centre
// (1e-7 e per cell: water10k forces 2e-7 off FP64 against 3e-8): it is summed
// in FP64.
template <int P>
__device__ __forceinline__ void sf_moments(const float4 *__restrict__ pk, uint32_t na, const ChebScale &cs, float4 s,
                                           float4 *__restrict__ s_at, float2 (&N)[P / 2], bool &beyond) {
  constexpr int B = cheb_b(P);
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int m = 0; m < P / 2; m++) N[m] = make_float2(0.f, 0.f);
  double charge = 0.0;
  float4 ahead = lane < na ? pk[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t b0 = 0; b0 < na; b0 += 32) {
    const uint32_t nb = min(32u, na - b0);
    float4 p = ahead;
    if (b0 + 32 + lane < na) ahead = pk[b0 + 32 + lane];
    else ahead = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool in = fmaf(p.x, p.x, fmaf(p.y, p.y, p.z * p.z)) <= cs.u2;
    beyond |= __any_sync(0xffffffffu, !in) != 0;
    p = in ? make_float4(p.x * cs.inv_u, p.y * cs.inv_u, p.z * cs.inv_u, p.w) : make_float4(0.f, 0.f, 0.f, 0.f);
    charge += (double)p.w;
    __syncwarp();
    s_at[lane] = p;
    __syncwarp();
#pragma unroll 4
    for (uint32_t j = 0; j < nb; j++) {
      const float4 a = s_at[j];
      const float x = fmaf(s.x, a.x, fmaf(s.y, a.y, s.z * a.z));
      const float x2 = x + x;
      float T[B + 1];
      T[0] = 1.0f;
      T[1] = x;
#pragma unroll
      for (int b = 2; b <= B; b++) T[b] = fmaf(x2, T[b - 1], -T[b - 2]);
      const float tb2 = T[B] + T[B];
      float g0 = a.w, g1 = a.w * T[B];
#pragma unroll
      for (int g = 0; g * B < P; g++) {
        const float2 gg = bcast(g0);
#pragma unroll
        for (int b = 0; b < B && g * B + b < P; b += 2)
          if (g == 0 && b == 0) N[0].y = fmaf(g0, x, N[0].y);
          else N[(g * B + b) / 2] = __ffma2_rn(gg, make_float2(T[b], T[b + 1]), N[(g * B + b) / 2]);
        const float g2 = fmaf(tb2, g1, -g0);
        g0 = g1;
        g1 = g2;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) charge += __shfl_xor_sync(0xffffffffu, charge, o);
  N[0].x = static_cast<float>(charge);
}

template <int P>
__device__ __forceinline__ void sf_tile(const SfArgs &a, const DirTile &u, const float4 *__restrict__ pk, uint32_t cnt,
                                        uint32_t cell, const float4 *rows, float4 *s_at, float2 *s_f) {
  const uint32_t lane = threadIdx.x & 31u;
  const float4 s = lane < u.n_dir ? a.dirs[u.dir_begin + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  const uint32_t node0 = u.node_begin - a.node_off;
  uint32_t a0 = 0;
  do {
    const uint32_t na = min((uint32_t)kSfAtomTile, cnt - a0);
    // few atoms: a sine and cosine per node cost 16 issue slots of the SFU,
    // the product P FMAs per node
    const bool series = P > 0 && 16u * na > (uint32_t)P;
    bool beyond = !series;
    float2 N[P > 0 ? P / 2 : 1];
    if constexpr (P > 0) {
      if (series) sf_moments<P>(pk + a0, na, a.cs, s, s_at, N, beyond);
    }
    for (uint32_t r0 = 0; r0 < u.n_rad; r0 += kSfRadChunk) {
      const uint32_t rc = min((uint32_t)kSfRadChunk, u.n_rad - r0);
      float2 *row = s_f + lane * sf_row(rc);
      __syncwarp();
      if (series) {
        if constexpr (P > 0) {
#pragma unroll 2
          for (uint32_t r = 0; r < rc; r++) {
            const float4 *t = rows + (size_t)(r0 + r) * (cheb_row(P) / 4);
            float2 f0 = make_float2(0.f, 0.f), f1 = make_float2(0.f, 0.f);
#pragma unroll
            for (int m = 0; m < cheb_row(P) / 4; m++) {
              const float4 c = t[m];
              f0 = __ffma2_rn(N[2 * m], make_float2(c.x, c.y), f0);
              if (2 * m + 1 < P / 2) f1 = __ffma2_rn(N[2 * m + 1], make_float2(c.z, c.w), f1);
            }
            row[r] = __fadd2_rn(f0, f1);
          }
        }
      } else {
        for (uint32_t r = 0; r < rc; r++) row[r] = make_float2(0.f, 0.f);
      }
      if (beyond && na) sf_direct(pk + a0, na, !series, a.cs.u2, s, a.kappa + u.kappa_begin + r0, rc, row);
      __syncwarp();
      // Coalesced stores: a whole direction's radial nodes are contiguous, so
      // with one chunk the tile's n_dir x n_rad nodes are one run; lanes are
      // aligned to the node blocks of S.
      if (rc == u.n_rad) {
        const uint32_t j0 = node0 % kNodeBlock;
        // m / rc by multiplication (m < 32 x 64), where rows are padded
        const uint32_t inv = sf_row(rc) == rc ? 0u : 0xffffffffu / rc + 1u;
        const uint32_t end = j0 + u.n_dir * rc;
        size_t o = ((size_t)(node0 / kNodeBlock) * a.ncell + cell) * kNodeBlock + lane;
        for (uint32_t k = lane; k < end; k += 32, o += (size_t)a.ncell * kNodeBlock) {
          if (k < j0) continue;
          const uint32_t m = k - j0;
          const float2 f = s_f[m + __umulhi(m, inv)];
          if (cnt <= kSfAtomTile) a.S[o] = f;
          else sf_store_dense(f, o, a0 > 0, a0 + kSfAtomTile >= cnt, a.S, a.lo_buf);
        }
      } else {
        for (uint32_t m = lane; m < u.n_dir * rc; m += 32) {
          const uint32_t d = m / rc, r = m - d * rc;
          const size_t o = sr_index(cell, node0 + d * u.n_rad + r0 + r, a.ncell);
          const float2 f = s_f[d * sf_row(rc) + r];
          if (cnt <= kSfAtomTile) a.S[o] = f;
          else sf_store_dense(f, o, a0 > 0, a0 + kSfAtomTile >= cnt, a.S, a.lo_buf);
        }
      }
    }
    a0 += kSfAtomTile;
  } while (a0 < cnt);
}

// Work item: kSfWarps consecutive tiles (of one group) and a.cells cells from
// `cell0` on.
__device__ __forceinline__ void sf_block(const SfArgs &a, uint32_t quad, uint32_t cell0) {
  extern __shared__ float4 s_sf[];
  const uint32_t warp = threadIdx.x >> 5;
  const DirTile u = a.tiles[quad * kSfWarps + warp];  // (a group's tiles are padded to whole quads)
  const uint32_t tab4 = u.n_rad * (uint32_t)(cheb_row((int)u.P) / 4);
  for (uint32_t i = threadIdx.x; i < tab4; i += kSfThreads) s_sf[i] = a.tab[u.tab / 4 + i];
  __syncthreads();
  if (u.n_dir == 0) return;
  const uint32_t rc = min(a.max_rad, (uint32_t)kSfRadChunk);
  float4 *s_at = s_sf + a.tab4 + warp * 32;
  float2 *s_f = reinterpret_cast<float2 *>(s_sf + a.tab4 + kSfWarps * 32) + (size_t)warp * 32 * sf_row(rc);
  const uint32_t cell1 = min(a.ncell, cell0 + a.cells);
#define GLST_SF_CASE(n)                                                                            \
  case n:                                                                                          \
    for (uint32_t cell = cell0; cell < cell1; cell++)                                              \
      sf_tile<n>(a, u, a.pk + a.cell_point[cell], a.cell_count[cell], cell, s_sf, s_at, s_f);      \
    break;
  switch (u.P) {
    GLST_SF_CASE(0) GLST_SF_CASE(4) GLST_SF_CASE(6) GLST_SF_CASE(8) GLST_SF_CASE(10)
    GLST_SF_CASE(12) GLST_SF_CASE(14) GLST_SF_CASE(16) GLST_SF_CASE(18) GLST_SF_CASE(20)
    GLST_SF_CASE(22) GLST_SF_CASE(24) GLST_SF_CASE(26) GLST_SF_CASE(28) GLST_SF_CASE(30)
    GLST_SF_CASE(32) GLST_SF_CASE(34) GLST_SF_CASE(36) GLST_SF_CASE(38) GLST_SF_CASE(40)
    GLST_SF_CASE(42) GLST_SF_CASE(44) GLST_SF_CASE(46) GLST_SF_CASE(48) GLST_SF_CASE(52)
    GLST_SF_CASE(56) GLST_SF_CASE(60) GLST_SF_CASE(64)
    default: break;
  }
#undef GLST_SF_CASE
}

__global__ void __launch_bounds__(kSfThreads, 4)
k_structure_factors(const __grid_constant__ SfArgs a, uint32_t cell_base) {
  const uint32_t quads = a.n_tiles / kSfWarps;
  const uint32_t c = blockIdx.x / quads;
  sf_block(a, blockIdx.x - c * quads, cell_base + c * a.cells);
}

// ----------------------------------------------------------------------------
// Shell sums (src/glst_force.cu:702-913 restated for shared memory): per
// node, an inclusive 3-D prefix sum of S over the cell grid (z, y, x), then
// R_c = w * [box(c, r_out) - box(c, r_in)], 8 corners per box, clipped to the
// grid.  All FP64.  Output R'_c(k) = R_c(k) e^{+ik.c} as float2, the twiddle
// built from per-axis tables e^{i kx cx} e^{i ky cy} e^{i kz cz}.
// CTA: nb nodes at once (rows of ncell+1 complex doubles in shared memory).
// (A form with a zero plane in front of each axis, so that corner offsets
// need no clipping tests, measured slower on water10k: 0.50 ms loading all
// eight corners of every box, 0.45 ms skipping the zero-plane corners,
// against 0.42 ms here -- the larger rows and their zeroing cost more than
// the index arithmetic saved.  Per-node tables of per-axis corner offsets,
// three shared loads per cell in place of the clipping arithmetic, measured
// slower too: 0.412 against 0.381 ms, a dependent shared load more per cell
// in a latency-bound loop.)
// Launch shapes: 512 threads, 3 CTAs per SM; 256 threads, 4 CTAs per SM
// where four CTAs' tables fit in shared memory (water10k, 8 nodes per CTA:
// 0.382 against 0.416 ms -- fewer threads per node give each thread more
// cells over which to spread its set-up, and four CTAs overlap their
// barrier-separated phases better; 4 nodes per CTA at any shape measured
// 0.55-0.66 ms); one node per CTA, 512 threads, on large grids (22^3 grid:
// 0.393 ms per 1,534 nodes against 0.399 with 1024 and 0.396 with 768
// threads; there the node's S loads and R stores, 8 bytes at a 256-byte
// stride in the node-block layout, take 25 % and 20 % of the time, the
// corners 19 %, the prefix passes 9 %).
constexpr int kSatThreads = 512;
constexpr int kSatThreadsSmall = 256;
constexpr int kSatThreadsOne = 512;  // one node per CTA (large grids)
// S loads in flight per thread: 8 (a 7-cell line in one batch on water10k),
// 4 in the 512-thread several-nodes form, whose register budget is 40 (8
// spilled there)
template <int kMinBlocks>
struct SatLoadBatch {
  static constexpr int value = kMinBlocks == 3 ? 4 : 8;
};

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

__device__ __forceinline__ double2 sat_at(const double2 *row, uint32_t x, uint32_t y,
                                          uint32_t z, const Grid &g) {
  return row[(x * g.ny + y) * g.nz + z];
}

__device__ __forceinline__ double2 cube_sum(const double2 *row, uint32_t x, uint32_t y,
                                            uint32_t z, uint32_t r, const Grid &g) {
  const uint32_t x0 = (x < r) ? 0 : x - r, y0 = (y < r) ? 0 : y - r, z0 = (z < r) ? 0 : z - r;
  const uint32_t x1 = min(x + r, g.nx - 1), y1 = min(y + r, g.ny - 1), z1 = min(z + r, g.nz - 1);
  const bool xb = x0 == 0, yb = y0 == 0, zb = z0 == 0;
  const uint32_t xm = xb ? 0 : x0 - 1, ym = yb ? 0 : y0 - 1, zm = zb ? 0 : z0 - 1;
  double2 s = sat_at(row, x1, y1, z1, g);
  double2 t;
  if (!xb) { t = sat_at(row, xm, y1, z1, g); s.x -= t.x; s.y -= t.y; }
  if (!yb) { t = sat_at(row, x1, ym, z1, g); s.x -= t.x; s.y -= t.y; }
  if (!zb) { t = sat_at(row, x1, y1, zm, g); s.x -= t.x; s.y -= t.y; }
  if (!xb && !yb) { t = sat_at(row, xm, ym, z1, g); s.x += t.x; s.y += t.y; }
  if (!xb && !zb) { t = sat_at(row, xm, y1, zm, g); s.x += t.x; s.y += t.y; }
  if (!yb && !zb) { t = sat_at(row, x1, ym, zm, g); s.x += t.x; s.y += t.y; }
  if (!xb && !yb && !zb) { t = sat_at(row, xm, ym, zm, g); s.x -= t.x; s.y -= t.y; }
  return s;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Dynamic shared memory: nb rows of `stride` complex (the SAT), the twiddle
// tables nb x (nx + ny + nz) complex, then, in the several-nodes form
// (kMinBlocks > 1, small grids) when it fits, the cell coordinates (ncell x
// u32, x | y << 10 | z << 20).  nb is a power of two <= 32: lane l of a warp works
// on node l % nb of the CTA and on the (l / nb)-th of the 32 / nb cells or
// lines the warp takes per step, so the per-node values (radii, weight,
// twiddle rows) stay in registers and the S loads and R stores of a warp are
// runs of consecutive nodes.
template <int kMinBlocks>
__device__ __forceinline__ void shell_block(const Grid &g, const SatArgs &a, uint32_t bx) {
  extern __shared__ double2 s_sat[];
  const uint32_t nb = a.nb, lg = a.lg_nb;
  const uint32_t k0 = bx * nb;
  const uint32_t C = g.ncell;
  const uint32_t naxis = g.nx + g.ny + g.nz;
  double2 *s_tw = s_sat + (size_t)nb * a.stride;
  uint32_t *s_xyz = reinterpret_cast<uint32_t *>(s_tw + (size_t)nb * naxis);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t j = lane & (nb - 1u);
  const uint32_t per_warp = 32u >> lg;
  const uint32_t first = warp * per_warp + (lane >> lg);
  const uint32_t step = (blockDim.x >> 5) * per_warp;
  const uint32_t k = k0 + j;         // node within the launch (node tables)
  const uint32_t ks = a.kbase + k;   // node within S and R
  const bool jv = k < a.K;
  // The S loads run as a flat sequence of batches (line l, z from z0) of
  // kLoadBatch cells each; the first is issued before the twiddle tables,
  // whose node loads and FP64 sincos it overlaps (water10k shell sums 0.441
  // vs 0.450 ms; one batch in flight ahead of the one summed, 0.462 ms at a
  // batch of 2 and spilling at 4).
  constexpr int kLoadBatch = SatLoadBatch<kMinBlocks>::value;
  const uint32_t nlines = g.nx * g.ny;
  const double2 zero = make_double2(0.0, 0.0);
  auto fetch = [&](float2 *dst, uint32_t line, uint32_t zb) {
#pragma unroll
    for (int u = 0; u < kLoadBatch; u++)
      dst[u] = (jv && line < nlines && zb + u < g.nz) ? __ldg(a.S + sr_index(line * g.nz + zb + u, ks, C))
                                                      : make_float2(0.f, 0.f);
  };
  float2 v[kLoadBatch];
  uint32_t l = first, z0 = 0;
  fetch(v, l, z0);
  // twiddle tables: e^{i k_a (i + 1/2) l} per node and axis
  for (uint32_t t = threadIdx.x; t < nb * naxis; t += blockDim.x) {
    const uint32_t jj = t / naxis, r = t - jj * naxis;
    const double4 nk = (k0 + jj < a.K) ? a.node64[k0 + jj] : make_double4(0.0, 0.0, 0.0, 0.0);
    double kc;
    if (r < g.nx) kc = nk.x * cell_centre(r, g.l);
    else if (r < g.nx + g.ny) kc = nk.y * cell_centre(r - g.nx, g.l);
    else kc = nk.z * cell_centre(r - g.nx - g.ny, g.l);
    double sn, cs;
    sincos(kc, &sn, &cs);
    s_tw[t] = make_double2(cs, sn);
  }
  auto coords = [&](uint32_t c) {
    const uint32_t x = c / (g.ny * g.nz), rem = c - x * (g.ny * g.nz);
    const uint32_t y = rem / g.nz, z = rem - y * g.nz;
    return x | (y << 10) | (z << 20);
  };
  if (kMinBlocks > 1 && a.xyz_table)
    for (uint32_t c = threadIdx.x; c < C; c += blockDim.x) s_xyz[c] = coords(c);
  double2 *row = s_sat + (size_t)j * a.stride;
  const double2 *twx = s_tw + (size_t)j * naxis, *twy = twx + g.nx, *twz = twy + g.ny;
  __syncthreads();  // twiddle tables
  // S[c][k0 + j] -> row j: the cell-relative structure factors times
  // e^{-ik.c} (the per-axis tables), summed along z on the way in (the z
  // prefix pass without its own shared-memory round trip)
  {
    double2 acc = zero, txy = zero;
    while (l < nlines) {
      uint32_t ln = l, zn = z0 + kLoadBatch;
      if (zn >= g.nz) { ln = l + step; zn = 0; }
      if (z0 == 0) {
        const uint32_t lx = l / g.ny;
        txy = cmul(twx[lx], twy[l - lx * g.ny]);  // e^{+i(kx cx + ky cy)}
        acc = zero;
      }
      const uint32_t base = l * g.nz;
#pragma unroll
      for (int u = 0; u < kLoadBatch; u++) {
        if (z0 + u < g.nz) {
          const double2 t = cmul(txy, twz[z0 + u]);  // e^{+ik.c}
          const double vx = v[u].x, vy = v[u].y;
          acc.x += vx * t.x + vy * t.y;  // v * conj(t)
          acc.y += vy * t.x - vx * t.y;
          row[base + z0 + u] = acc;
        }
      }
      fetch(v, ln, zn);
      l = ln;
      z0 = zn;
    }
  }
  __syncthreads();
  // prefix along y (lines x, z)
  for (uint32_t l = first; l < g.nx * g.nz; l += step) {
    const uint32_t x = l / g.nz, z = l - x * g.nz;
    double2 *p = row + x * g.ny * g.nz + z;
    double2 acc = make_double2(0.0, 0.0);
    for (uint32_t y = 0; y < g.ny; y++) { acc.x += p[y * g.nz].x; acc.y += p[y * g.nz].y; p[y * g.nz] = acc; }
  }
  __syncthreads();
  // prefix along x (lines y, z)
  {
    const uint32_t sx = g.ny * g.nz;
    for (uint32_t l = first; l < sx; l += step) {
      double2 *p = row + l;
      double2 acc = make_double2(0.0, 0.0);
      for (uint32_t x = 0; x < g.nx; x++) { acc.x += p[x * sx].x; acc.y += p[x * sx].y; p[x * sx] = acc; }
    }
  }
  __syncthreads();
  if (!jv) return;
  // shell sums, weight and twiddle
  const uint32_t radii = a.node_radii[k];
  const uint32_t r_out = radii >> 16, r_in = radii & 0xffffu;
  const double w = a.node64[k].w;
  // The thread's cells c = first + i * step.  Small grids (several nodes per
  // CTA) look their coordinates up in the CTA's table.  Large grids (one node
  // per CTA) step them with carries: there the table cost every CTA two
  // divisions per cell of the grid (water333k shell sums 34.8 ms with it,
  // 27.9 ms stepping); on small grids stepping measured slower (water10k
  // 0.43 against 0.42 ms).
  if constexpr (kMinBlocks > 1) {
    for (uint32_t c = first; c < C; c += step) {
      const uint32_t xyz = a.xyz_table ? s_xyz[c] : coords(c);
      const uint32_t x = xyz & 1023u, y = (xyz >> 10) & 1023u, z = xyz >> 20;
      const double2 o = cube_sum(row, x, y, z, r_out, g);
      const double2 i = cube_sum(row, x, y, z, r_in, g);
      const double2 sh = make_double2((o.x - i.x) * w, (o.y - i.y) * w);
      const double2 r = cmul(cmul(sh, twx[x]), cmul(twy[y], twz[z]));
      a.R[sr_index(c, ks, C)] = make_float2(static_cast<float>(r.x), static_cast<float>(r.y));
    }
  } else {
    const uint32_t syz = g.ny * g.nz;
    const uint32_t sx = step / syz, sy = (step - sx * syz) / g.nz, sz = step - sx * syz - sy * g.nz;
    uint32_t x = first / syz, y = (first - x * syz) / g.nz, z = first - x * syz - y * g.nz;
    for (uint32_t c = first; c < C; c += step) {
      const double2 o = cube_sum(row, x, y, z, r_out, g);
      const double2 i = cube_sum(row, x, y, z, r_in, g);
      const double2 sh = make_double2((o.x - i.x) * w, (o.y - i.y) * w);
      const double2 r = cmul(cmul(sh, twx[x]), cmul(twy[y], twz[z]));
      a.R[sr_index(c, ks, C)] = make_float2(static_cast<float>(r.x), static_cast<float>(r.y));
      z += sz;  // sz < nz and sy < ny: one carry at most per axis
      if (z >= g.nz) { z -= g.nz; y++; }
      y += sy;
      if (y >= g.ny) { y -= g.ny; x++; }
      x += sx;
    }
  }
}

template <int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
k_shell_sums(Grid g, SatArgs a) {
  shell_block<kMinBlocks>(g, a, blockIdx.x);
}

// ----------------------------------------------------------------------------
// Shell sums for grids whose per-node prefix table does not fit in shared
// memory (the same arithmetic as k_shell_sums, src/glst_force.cu:702-913):
// the FP64 summed-area tables of a batch of node blocks live in global memory
// (laid out like S: per block of kNodeBlock nodes, cell-major, node fastest,
// so every warp access is a contiguous run of 32 nodes), built by three
// line passes (z with the twiddle e^{-ik.c} applied on load, then y, then x)
// and read by a fourth pass that forms the 16-corner shell differences.  The
// per-axis twiddles of the stage's nodes are tabulated once per stage.
struct GsatArgs {
  const float2 *S;              // stage-local structure factors
  const double4 *node64;        // node table of the stage (kx, ky, kz, w)
  const uint32_t *node_radii;   // r_in | r_out << 16, same indexing
  const double2 *tw;            // twiddles e^{+i k_a c_a}: tw[a * K + k], a = 0 .. nx + ny + nz - 1
  double2 *T;                   // tables of the batch: nblk x C x kNodeBlock
  float2 *R;                    // stage-local shell sums
  uint32_t K;                   // nodes of the stage
  uint32_t blk0;                // first node block of the batch (stage-local)
  uint32_t nblk;                // node blocks in the batch
};

// Twiddle table: tw[a * K + k] = e^{+i k_axis (i + 1/2) l} for the a-th of
// the nx + ny + nz per-axis cell indices (node fastest, so the warps of the
// passes, 32 consecutive nodes each, read contiguous runs).
__global__ void k_gsat_twiddles(Grid g, const double4 *__restrict__ node64, uint32_t K,
                                double2 *__restrict__ tw) {
  const uint32_t naxis = g.nx + g.ny + g.nz;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)K * naxis) return;
  const uint32_t r = (uint32_t)(t / K), k = (uint32_t)(t - (size_t)r * K);
  const double4 nk = node64[k];
  double kc;
  if (r < g.nx) kc = nk.x * cell_centre(r, g.l);
  else if (r < g.nx + g.ny) kc = nk.y * cell_centre(r - g.nx, g.l);
  else kc = nk.z * cell_centre(r - g.nx - g.ny, g.l);
  double sn, cs;
  sincos(kc, &sn, &cs);
  tw[t] = make_double2(cs, sn);
}

__device__ __forceinline__ size_t gsat_at(uint32_t bb, uint32_t c, uint32_t j, uint32_t C) {
  return ((size_t)bb * C + c) * kNodeBlock + j;
}

// Pass 1: thread = (line (x, y), block, node j); S x e^{-ik.c}, prefix along z.
__global__ void k_gsat_z(Grid g, GsatArgs a) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t j = (uint32_t)(t % kNodeBlock);
  const size_t lb = t / kNodeBlock;
  const uint32_t bb = (uint32_t)(lb % a.nblk);
  const size_t line = lb / a.nblk;
  if (line >= (size_t)g.nx * g.ny) return;
  const uint32_t blk = a.blk0 + bb;
  const uint32_t k = blk * kNodeBlock + j;  // stage-local node
  const uint32_t C = g.ncell;
  const uint32_t x = (uint32_t)(line / g.ny), y = (uint32_t)(line - (size_t)x * g.ny);
  const uint32_t c0 = (uint32_t)line * g.nz;
  double2 *T = a.T;
  if (k >= a.K) {
    for (uint32_t z = 0; z < g.nz; z++) T[gsat_at(bb, c0 + z, j, C)] = make_double2(0.0, 0.0);
    return;
  }
  const size_t K = a.K;
  const double2 *tk = a.tw + k;  // entry of axis index i: tk[i * K]
  const double2 txy = cmul(tk[(size_t)x * K], tk[(size_t)(g.nx + y) * K]);
  const double2 *twz = tk + (size_t)(g.nx + g.ny) * K;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (uint32_t z = 0; z < g.nz; z++) {
    const float2 v = a.S[sr_index(c0 + z, k, C)];
    const double2 tt = cmul(txy, twz[(size_t)z * K]);
    const double vx = v.x, vy = v.y;
    acc.x += vx * tt.x + vy * tt.y;  // v * conj(tt)
    acc.y += vy * tt.x - vx * tt.y;
    T[gsat_at(bb, c0 + z, j, C)] = acc;
  }
}

// Passes 2 and 3: prefix along y (axis 1) or x (axis 0), in place.
__global__ void k_gsat_prefix(Grid g, GsatArgs a, int axis) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t j = (uint32_t)(t % kNodeBlock);
  const size_t lb = t / kNodeBlock;
  const uint32_t bb = (uint32_t)(lb % a.nblk);
  const size_t line = lb / a.nblk;
  const uint32_t C = g.ncell;
  uint32_t n, c0, stride;
  if (axis == 1) {  // lines (x, z)
    if (line >= (size_t)g.nx * g.nz) return;
    const uint32_t x = (uint32_t)(line / g.nz), z = (uint32_t)(line - (size_t)x * g.nz);
    n = g.ny; c0 = x * g.ny * g.nz + z; stride = g.nz;
  } else {  // lines (y, z)
    if (line >= (size_t)g.ny * g.nz) return;
    n = g.nx; c0 = (uint32_t)line; stride = g.ny * g.nz;
  }
  double2 *T = a.T;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (uint32_t i = 0; i < n; i++) {
    double2 *p = T + gsat_at(bb, c0 + i * stride, j, C);
    const double2 v = *p;
    acc.x += v.x;
    acc.y += v.y;
    *p = acc;
  }
}

__device__ __forceinline__ double2 gcube_sum(const double2 *T, uint32_t bb, uint32_t j, uint32_t x, uint32_t y,
                                             uint32_t z, uint32_t r, const Grid &g) {
  const uint32_t C = g.ncell;
  const uint32_t x0 = (x < r) ? 0 : x - r, y0 = (y < r) ? 0 : y - r, z0 = (z < r) ? 0 : z - r;
  const uint32_t x1 = min(x + r, g.nx - 1), y1 = min(y + r, g.ny - 1), z1 = min(z + r, g.nz - 1);
  const bool xb = x0 == 0, yb = y0 == 0, zb = z0 == 0;
  const uint32_t xm = xb ? 0 : x0 - 1, ym = yb ? 0 : y0 - 1, zm = zb ? 0 : z0 - 1;
  auto at = [&](uint32_t a, uint32_t b, uint32_t c) { return T[gsat_at(bb, (a * g.ny + b) * g.nz + c, j, C)]; };
  double2 s = at(x1, y1, z1);
  double2 t;
  if (!xb) { t = at(xm, y1, z1); s.x -= t.x; s.y -= t.y; }
  if (!yb) { t = at(x1, ym, z1); s.x -= t.x; s.y -= t.y; }
  if (!zb) { t = at(x1, y1, zm); s.x -= t.x; s.y -= t.y; }
  if (!xb && !yb) { t = at(xm, ym, z1); s.x += t.x; s.y += t.y; }
  if (!xb && !zb) { t = at(xm, y1, zm); s.x += t.x; s.y += t.y; }
  if (!yb && !zb) { t = at(x1, ym, zm); s.x += t.x; s.y += t.y; }
  if (!xb && !yb && !zb) { t = at(xm, ym, zm); s.x -= t.x; s.y -= t.y; }
  return s;
}

// Pass 4: thread = (cell, block, node j): shell difference x w x e^{+ik.c}.
__global__ void k_gsat_shell(Grid g, GsatArgs a) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t j = (uint32_t)(t % kNodeBlock);
  const size_t cb = t / kNodeBlock;
  const uint32_t bb = (uint32_t)(cb % a.nblk);
  const size_t c = cb / a.nblk;
  if (c >= g.ncell) return;
  const uint32_t k = (a.blk0 + bb) * kNodeBlock + j;
  if (k >= a.K) return;
  const uint32_t syz = g.ny * g.nz;
  const uint32_t x = (uint32_t)(c / syz), rem = (uint32_t)(c - (size_t)x * syz);
  const uint32_t y = rem / g.nz, z = rem - y * g.nz;
  const uint32_t radii = a.node_radii[k];
  const uint32_t r_out = radii >> 16, r_in = radii & 0xffffu;
  const double w = a.node64[k].w;
  const double2 o = gcube_sum(a.T, bb, j, x, y, z, r_out, g);
  const double2 i = gcube_sum(a.T, bb, j, x, y, z, r_in, g);
  const double2 sh = make_double2((o.x - i.x) * w, (o.y - i.y) * w);
  const size_t K = a.K;
  const double2 *tk = a.tw + k;
  const double2 r = cmul(cmul(sh, tk[(size_t)x * K]), cmul(tk[(size_t)(g.nx + y) * K], tk[(size_t)(g.nx + g.ny + z) * K]));
  a.R[sr_index((uint32_t)c, k, g.ncell)] = make_float2(static_cast<float>(r.x), static_cast<float>(r.y));
}

// ----------------------------------------------------------------------------
// Long-range gather (src/glst_force.cu:983-1135 restated):
//   en_i = q_i Re sum_k e^{ik.d_i} R'_c(k),   f_i = q_i sum_k Im(...) k.
// Per direction s_j the sum over its radial nodes is a function of u = s_j.d_i
// alone, and with the series of the structure factors a short one:
//   e(x) = Re sum_r e^{i kappa_r U x} R'_r = sum_p c_p T_p(x),   x = u / U,
//   c_p = sum_r (2 - [p = 0]) Re(i^p R'_r) J_p(kappa_r U),
//   sum_r kappa_r Im(e^{i kappa_r u} R'_r) = -e'(x) / U.
// The weights in R' (a Gaussian in kappa) let fewer terms do than the
// structure factors need: P = 30, 18 and 14 in water10k's groups.  So a
// (cell, direction) takes one n_rad x P product, and an (atom, direction) two
// short series instead of a sine, a cosine and six FMAs per node (water10k
// 1.40 ms, at the SFU's bound).
//
// Lane = direction, atoms broadcast from shared memory: both series'
// coefficients stay in registers as (e, e') pairs for paired FP32
// instructions, and the inner loop loads nothing but the atom.  In the
// product basis T_{Bg} T_b the inner sums over b need B - 1 Chebyshev values
// and the outer sum over g another P / B.  The 32 directions are then summed
// across the warp for eight atoms at a time: 31 shuffles leave one of the 8 x
// 4 sums in each lane.  FP32 over the 32 directions, FP64 across direction
// tiles and warps.  Atoms beyond the series' range and tiles of too few atoms
// for the product take a sine and cosine per node (lr_direct).
//
// Warps are independent: each takes a cell and a chunk of direction tiles,
// with no CTA barriers (four warps on one cell's chunk waited for each other
// a third of the time).  A tile's R' is copied to shared memory
// asynchronously while the previous tile's series are evaluated -- the buffer
// is free once its coefficients are formed.  The groups' tables are copied to
// shared memory where three CTAs per SM still fit with them (water10k 485 ->
// 478 us, 168 atoms per cell 149 -> 143, 648 atoms 47 -> 42).
// Measured: water10k 1.458 -> 0.485 ms, 3,000 atoms on 4^3 cells 0.141 ->
// 0.076 ms, 168 atoms per cell 0.279 -> 0.148 ms, a million atoms 55 -> 17 ms;
// forces 1.5e-8 -> 0.9e-8 off the FP64 path.
constexpr int kLrWarps = 4;
constexpr int kLrThreads = 32 * kLrWarps;
constexpr int kLrAtomTile = 128;
constexpr int kLrBatch = 8;       // atoms reduced across the warp together
constexpr uint32_t kLrMaxRad = 256;    // radial nodes per direction, at most (set-up checks)
constexpr uint32_t kLrMaxQuads = 128;  // radial nodes of all groups, in fours, at most (set-up checks)

struct LrArgs {
  const float4 *pk;
  const uint32_t *cell_count, *cell_point;
  const DirTile *tiles;
  const float4 *dirs;
  const float *kappa;
  const float4 *tab;   // Chebyshev series, cheb_row(P) floats per radial node
  const float2 *R;
  double4 *part;       // one row of natom per chunk of tiles
  ChebScale cs;
  uint32_t ncell, n_tiles, tiles_per_chunk, max_rad, node_off, natom;
  int accumulate;      // a later node stage adds into the same rows
  uint32_t tab4;       // float4s of all groups' tables
};

__host__ __device__ inline size_t lr_smem_bytes(uint32_t max_rad) {
  const uint32_t rc = max_rad < (uint32_t)kSfRadChunk ? max_rad : (uint32_t)kSfRadChunk;
  return (size_t)kLrWarps * (kLrAtomTile * (sizeof(float4) + 4 * sizeof(double)) + 32 * sf_row(rc) * sizeof(float2));
}

// The general form for a warp's 32 directions: the tile's atoms beyond the
// series' range (all: every atom), one sine and cosine per (atom, node).
__device__ __noinline__ void lr_direct(const LrArgs &a, const DirTile &u, const float4 *__restrict__ atoms,
                                       uint32_t na, bool all, uint32_t cell, double *__restrict__ acc) {
  const uint32_t lane = threadIdx.x & 31u;
  const bool act = lane < u.n_dir;
  const float4 s = act ? a.dirs[u.dir_begin + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  const uint32_t node0 = u.node_begin - a.node_off + (act ? lane : 0) * u.n_rad;
  for (uint32_t j = 0; j < na; j++) {
    const float4 p = atoms[j];
    if (!all && fmaf(p.x, p.x, fmaf(p.y, p.y, p.z * p.z)) <= a.cs.u2) continue;
    const float x = fmaf(s.x, p.x, fmaf(s.y, p.y, s.z * p.z));
    float e = 0.f, g = 0.f;
    for (uint32_t r = 0; r < u.n_rad; r++) {
      const float kap = a.kappa[u.kappa_begin + r];
      const float2 v = a.R[sr_index(cell, node0 + r, a.ncell)];
      float sn, cs, sg;
      fma_sincos_signed(kap * x, 1.0f, &sn, &cs, &sg);
      e = fmaf(sg, fmaf(cs, v.x, -sn * v.y), e);
      g = fmaf(kap * sg, fmaf(cs, v.y, sn * v.x), g);
    }
    if (!act) e = g = 0.f;
    float f[4] = {e, g * s.x, g * s.y, g * s.z};
#pragma unroll
    for (int c = 0; c < 4; c++)
      for (int o = 16; o > 0; o >>= 1) f[c] += __shfl_xor_sync(0xffffffffu, f[c], o);
    if (lane < 4) acc[4 * j + lane] += (double)(lane == 0 ? f[0] : lane == 1 ? f[1] : lane == 2 ? f[2] : f[3]);
  }
}

// Sum two atoms' values over lanes that differ in `bit`: lanes with the bit
// clear keep the first atom's, the others the second's.
template <int NV>
__device__ __forceinline__ void lr_merge(const float *a, const float *b, int bit, float *out) {
  const bool up = (threadIdx.x & bit) != 0;
#pragma unroll
  for (int c = 0; c < NV; c++) {
    const float keep = up ? b[c] : a[c], give = up ? a[c] : b[c];
    out[c] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
  }
}

// One direction's two series at a scaled atom: (e, e').
template <int P>
__device__ __forceinline__ float2 lr_series(const float2 (&AB)[P], float4 s, float4 at) {
  constexpr int B = cheb_b(P);
  const float x = fmaf(s.x, at.x, fmaf(s.y, at.y, s.z * at.z));
  const float x2 = x + x;
  float T[B + 1];
  T[0] = 1.0f;
  T[1] = x;
#pragma unroll
  for (int b = 2; b <= B; b++) T[b] = fmaf(x2, T[b - 1], -T[b - 2]);
  const float tb2 = T[B] + T[B];
  float g0 = 1.0f, g1 = T[B];
  float2 sum = make_float2(0.f, 0.f);
#pragma unroll
  for (int g = 0; g * B < P; g++) {
    float2 in = AB[g * B];
#pragma unroll
    for (int b = 1; b < B && g * B + b < P; b++) in = __ffma2_rn(AB[g * B + b], bcast(T[b]), in);
    sum = g == 0 ? in : __ffma2_rn(in, bcast(g0), sum);
    const float g2 = fmaf(tb2, g1, -g0);
    g0 = g1;
    g1 = g2;
  }
  return sum;
}

// R' of a tile whose radial nodes fit one chunk, to shared memory, without
// waiting: the tile's nodes are one run, lanes aligned to R's node blocks.
__device__ __forceinline__ void lr_fetch(const LrArgs &a, const DirTile &u, uint32_t cell, float2 *s_r) {
  const uint32_t lane = threadIdx.x & 31u, rc = u.n_rad;
  if (rc <= (uint32_t)kSfRadChunk) {
    const uint32_t node0 = u.node_begin - a.node_off, j0 = node0 % kNodeBlock;
    const uint32_t inv = sf_row(rc) == rc ? 0u : 0xffffffffu / rc + 1u;
    const uint32_t end = j0 + u.n_dir * rc;
    const float2 *src = a.R + ((size_t)(node0 / kNodeBlock) * a.ncell + cell) * kNodeBlock + lane;
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(s_r));
    for (uint32_t k = lane; k < end; k += 32, src += (size_t)a.ncell * kNodeBlock)
      if (k >= j0) {
        const uint32_t m = k - j0 + __umulhi(k - j0, inv);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8u * m), "l"(src) : "memory");
      }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// One tile's series at the warp's na atoms, added to acc.  `next`: the tile
// whose R' is fetched meanwhile (if any).
template <int P, bool kTabShared>
__device__ __forceinline__ void lr_tile(const LrArgs &a, const DirTile &u, const DirTile *next, uint32_t na,
                                        uint32_t cell, const float4 *__restrict__ s_at, double *__restrict__ acc,
                                        float2 *s_r) {
  constexpr int B = cheb_b(P);
  const uint32_t lane = threadIdx.x & 31u;
  const float4 s = lane < u.n_dir ? a.dirs[u.dir_begin + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
  float2 c2[P / 2];  // (c_p, c_{p+1})
#pragma unroll
  for (int m = 0; m < P / 2; m++) c2[m] = make_float2(0.f, 0.f);
  for (uint32_t r0 = 0; r0 < u.n_rad; r0 += kSfRadChunk) {
    const uint32_t rc = min((uint32_t)kSfRadChunk, u.n_rad - r0);
    if (rc < u.n_rad) {
      const uint32_t node0 = u.node_begin - a.node_off;
      __syncwarp();
      for (uint32_t m = lane; m < u.n_dir * rc; m += 32) {
        const uint32_t d = m / rc, r = m - d * rc;
        s_r[d * sf_row(rc) + r] = a.R[sr_index(cell, node0 + d * u.n_rad + r0 + r, a.ncell)];
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    const float2 *row = s_r + (lane < u.n_dir ? lane : 0) * sf_row(rc);
    extern __shared__ float4 s_lr[];
    const float4 *t = (kTabShared ? s_lr : a.tab) + u.lr_tab / 4 + (size_t)r0 * (cheb_row(P) / 4);
#pragma unroll 2
    for (uint32_t r = 0; r < rc; r++, t += cheb_row(P) / 4) {
      const float2 v = row[r];
#pragma unroll
      for (int m = 0; m < cheb_row(P) / 4; m++) {
        const float4 c = kTabShared ? t[m] : __ldg(t + m);
        c2[2 * m] = __ffma2_rn(v, make_float2(c.x, c.y), c2[2 * m]);
        if (2 * m + 1 < P / 2) c2[2 * m + 1] = __ffma2_rn(v, make_float2(c.z, c.w), c2[2 * m + 1]);
      }
    }
  }
  __syncwarp();  // every lane has read its row
  if (next) lr_fetch(a, *next, cell, s_r);
  // (c_p, c'_p): the derivative's series by c'_{p-1} = c'_{p+1} + 2 p c_p,
  // then both in the product basis (T_{Bg+b} = 2 T_{Bg} T_b - T_{Bg-b})
  float2 AB[P];
#pragma unroll
  for (int p = 0; p < P; p++) AB[p].x = (p & 1) ? c2[p / 2].y : c2[p / 2].x;
  AB[P - 1].y = 0.f;
#pragma unroll
  for (int p = P - 1; p > 0; p--) AB[p - 1].y = fmaf(2.0f * p, AB[p].x, p + 1 < P ? AB[p + 1].y : 0.f);
  AB[0].y *= 0.5f;
#pragma unroll
  for (int p = P - 1; p > B; p--) {
    const int g = p / B, b = p % B;
    if (b == 0) continue;
    AB[B * g - b] = __ffma2_rn(AB[p], bcast(-1.0f), AB[B * g - b]);
    AB[p] = __fadd2_rn(AB[p], AB[p]);
  }
  // inactive lanes contribute nothing
  const float live = lane < u.n_dir ? 1.0f : 0.0f;
  // g = -e' / U
  const float3 sg = make_float3(-a.cs.inv_u * s.x, -a.cs.inv_u * s.y, -a.cs.inv_u * s.z);
  const uint32_t slot = 4u * (((lane >> 4) & 1u) + 2u * ((lane >> 3) & 1u) + 4u * ((lane >> 2) & 1u)) + (lane & 3u);
  for (uint32_t j0 = 0; j0 < na; j0 += kLrBatch) {
    float q4[2][4];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float m2[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        float v[2][4];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const float2 eg = lr_series<P>(AB, s, s_at[j0 + 4 * h + 2 * i + k]);
          v[k][0] = live * eg.x;
          v[k][1] = eg.y * sg.x;
          v[k][2] = eg.y * sg.y;
          v[k][3] = eg.y * sg.z;
        }
        lr_merge<4>(v[0], v[1], 16, m2[i]);
      }
      lr_merge<4>(m2[0], m2[1], 8, q4[h]);
    }
    float e4[4], e2[2], e1[1];
    lr_merge<4>(q4[0], q4[1], 4, e4);
    lr_merge<2>(e4, e4 + 2, 2, e2);
    lr_merge<1>(e2, e2 + 1, 1, e1);
    acc[4 * j0 + slot] += (double)e1[0];
  }
}

// Work item of a warp: a cell and a chunk of direction tiles.
template <bool kTabShared>
__device__ __forceinline__ void lr_warp(const LrArgs &a, uint32_t cell, uint32_t chunk) {
  extern __shared__ float4 s_lr[];
  const uint32_t cnt = a.cell_count[cell];
  if (cnt == 0) return;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t start = a.cell_point[cell];
  const uint32_t t0 = chunk * a.tiles_per_chunk, t1 = min(a.n_tiles, t0 + a.tiles_per_chunk);
  const uint32_t rc = min(a.max_rad, (uint32_t)kSfRadChunk);
  float4 *s_own = s_lr + (kTabShared ? a.tab4 : 0u);  // (the tables come first)
  float4 *s_at = s_own + warp * kLrAtomTile;
  double *acc = reinterpret_cast<double *>(s_own + kLrWarps * kLrAtomTile) + warp * (kLrAtomTile * 4);
  float2 *s_r = reinterpret_cast<float2 *>(reinterpret_cast<double *>(s_own + kLrWarps * kLrAtomTile) +
                                           kLrWarps * kLrAtomTile * 4) + (size_t)warp * 32 * sf_row(rc);
  for (uint32_t a0 = 0; a0 < cnt; a0 += kLrAtomTile) {
    const uint32_t na = min((uint32_t)kLrAtomTile, cnt - a0), pad = (na + kLrBatch - 1) & ~(uint32_t)(kLrBatch - 1);
    // the first series tile
    auto is_series = [&](const DirTile &u) { return u.n_dir > 0 && u.lr_P > 0 && 16u * na > u.lr_P; };
    uint32_t t = t0;
    while (t < t1 && !is_series(a.tiles[t])) t++;
    DirTile u;
    if (t < t1) {
      u = a.tiles[t];
      lr_fetch(a, u, cell, s_r);
    }
    bool beyond = false;
    for (uint32_t i = lane; i < 4 * pad; i += 32) acc[i] = 0.0;
    for (uint32_t b0 = 0; b0 < pad; b0 += 32) {
      const uint32_t i = b0 + lane;
      const float4 p = i < na ? a.pk[start + a0 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const bool in = fmaf(p.x, p.x, fmaf(p.y, p.y, p.z * p.z)) <= a.cs.u2;
      // (an atom beyond the range: its series sums are dropped below)
      s_at[i] = in ? make_float4(p.x * a.cs.inv_u, p.y * a.cs.inv_u, p.z * a.cs.inv_u, 0.f)
                   : make_float4(0.f, 0.f, 0.f, 1.f);
      beyond |= __any_sync(0xffffffffu, !in) != 0;
    }
    __syncwarp();
    while (t < t1) {
      uint32_t tn = t + 1;
      while (tn < t1 && !is_series(a.tiles[tn])) tn++;
      DirTile un;
      if (tn < t1) un = a.tiles[tn];
      const DirTile *next = tn < t1 ? &un : nullptr;
#define GLST_LR_CASE(n) \
  case n: lr_tile<n, kTabShared>(a, u, next, na, cell, s_at, acc, s_r); break;
      switch (u.lr_P) {
      GLST_LR_CASE(4) GLST_LR_CASE(6) GLST_LR_CASE(8) GLST_LR_CASE(10) GLST_LR_CASE(12)
      GLST_LR_CASE(14) GLST_LR_CASE(16) GLST_LR_CASE(18) GLST_LR_CASE(20) GLST_LR_CASE(22)
      GLST_LR_CASE(24) GLST_LR_CASE(26) GLST_LR_CASE(28) GLST_LR_CASE(30) GLST_LR_CASE(32)
      GLST_LR_CASE(34) GLST_LR_CASE(36) GLST_LR_CASE(38) GLST_LR_CASE(40) GLST_LR_CASE(42)
      GLST_LR_CASE(44) GLST_LR_CASE(46) GLST_LR_CASE(48) GLST_LR_CASE(52) GLST_LR_CASE(56)
      GLST_LR_CASE(60) GLST_LR_CASE(64)
        default: break;
      }
#undef GLST_LR_CASE
      t = tn;
      u = un;
    }
    __syncwarp();
    if (beyond) {  // drop their series sums; lr_direct gives theirs
      for (uint32_t i = lane; i < na; i += 32)
        if (s_at[i].w != 0.f) acc[4 * i] = acc[4 * i + 1] = acc[4 * i + 2] = acc[4 * i + 3] = 0.0;
      __syncwarp();
    }
    for (uint32_t td = t0; td < t1; td++) {
      const DirTile d = a.tiles[td];
      if (d.n_dir == 0) continue;
      const bool series = is_series(d);
      if (!series || beyond) lr_direct(a, d, a.pk + start + a0, na, !series, cell, acc);
    }
    __syncwarp();
    for (uint32_t i = lane; i < na; i += 32) {
      const double q = static_cast<double>(a.pk[start + a0 + i].w);
      double4 *dst = a.part + (size_t)chunk * a.natom + start + a0 + i;
      double4 o = make_double4(q * acc[4 * i + 1], q * acc[4 * i + 2], q * acc[4 * i + 3], q * acc[4 * i]);
      if (a.accumulate) {
        const double4 d = *dst;
        o = make_double4(d.x + o.x, d.y + o.y, d.z + o.z, d.w + o.w);
      }
      *dst = o;
    }
    __syncwarp();
  }
}

// Items chunk by chunk, so that the first (largest) groups' work starts first
// and a CTA's warps share a chunk's tables.
template <bool kTabShared>
__global__ void __launch_bounds__(kLrThreads, 3)
k_long_range(const __grid_constant__ LrArgs a, uint32_t n_chunks) {
  if constexpr (kTabShared) {
    extern __shared__ float4 s_lr[];
    for (uint32_t i = threadIdx.x; i < a.tab4; i += kLrThreads) s_lr[i] = a.tab[i];
    __syncthreads();
  }
  const uint64_t item = (uint64_t)blockIdx.x * kLrWarps + (threadIdx.x >> 5);
  const uint32_t chunk = (uint32_t)(item / a.ncell);
  if (chunk >= n_chunks) return;
  lr_warp<kTabShared>(a, (uint32_t)(item - (uint64_t)chunk * a.ncell), chunk);
}

// ----------------------------------------------------------------------------
// Near field (src/glst_force.cu:1170-1544 restated): bare q_i q_j / r over
// the own cell (self skipped) and the up to 26 neighbour cells inside the
// grid (open boundary).  FP64 throughout, bound by the FP64 pipe: 20
// operations per pair, the reciprocal square root a hardware approximation
// and two Newton steps (below) instead of the library's general one.
//
// The three neighbour cells along z are consecutive cells, so their atoms are
// one run: nine runs, (dx, dy), cover the neighbourhood.  One warp per (32
// atoms of a cell, row of runs), the runs' atoms staged 32 at a time in the
// warp's own shared memory, the next 32 loaded meanwhile -- no CTA barriers,
// and full batches where cells hold few atoms.  Cells of at most 16 or 8 atoms
// split each batch over two or four groups of lanes, and so do systems too
// small to fill the GPU with one lane per (atom, row) (sr_width).  A row is one run or the
// three of an x plane, and writes its own partial row of per-atom sums, summed
// by k_combine in a fixed order.
// Measured (one thread per atom and CTA barriers between cells before):
// water10k 0.291 -> 0.220 ms, 168 atoms per cell 0.400 -> 0.285 ms, 26^3 cells
// of 6 atoms 0.485 -> 0.101 ms, 3,000 atoms on 4^3 cells 0.067 -> 0.052 ms, a
// million atoms 4.44 -> 4.03 ms.
constexpr int kSrThreads = 128;
constexpr int kSrWarps = kSrThreads / 32;
constexpr int kSrRowsPlanes = 3;
constexpr int kSrRowsLines = 9;
constexpr int kSrRowsMax = kSrRowsLines;

// 1 / sqrt(x) by Newton's method (the Newton-Raphson iteration for the root of
// 1 / y^2 - x: y <- y (3 - x y^2) / 2), twice, from the hardware's
// approximation.  A relative error d becomes 3 d^2 / 2, so a start within 2^-15
// leaves less than 1e-17 after two steps; what remains is rounding, at most
// 1.5 x 2^-53 (half of it of x y^2 in the second step's residual, 2^-53 of the
// result).  Zero, infinity and not-a-number give the approximation, which is
// CUDA's rsqrt of them; squares below the smallest normal number count as zero.
// Measured against CUDA's rsqrt: near field of 30,000 atoms on 7^3 cells 166
// against 191 us, 21,000 atoms on 5^3 cells 191 against 219, 100,000 atoms on
// 26^3 cells 97 against 122.
__device__ __forceinline__ double sr_rsqrt(double x) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
  const double hx = 0.5 * x;
  const double y1 = y0 * fma(-hx * y0, y0, 1.5);
  const double y = fma(fma(-hx * y1, y1, 0.5), y1, y1);
  return (__double2hiint(y) & 0x7fffffff) < 0x7ff00000 ? y : y0;
}

struct SrSum {
  double x, y, z, e;
};

// One staged batch: lanes take atoms sub, sub + groups, ..., four at a time in
// four independent chains (a pair is a dozen dependent FP64 operations, and
// their latency, not their number, bounds a warp that does one pair after
// another).  The batch is padded with uncharged far-away atoms.
constexpr int kSrChains = 4;
template <bool kOwn>
__device__ __forceinline__ void sr_batch(const double4 *s_at, uint32_t n, uint32_t sub, uint32_t groups,
                                         const double4 &me, uint32_t self, SrSum (&f)[kSrChains]) {
#pragma unroll 1
  for (uint32_t j0 = sub; j0 < n; j0 += kSrChains * groups) {
    double dx[kSrChains], dy[kSrChains], dz[kSrChains], ir[kSrChains], q[kSrChains];
#pragma unroll
    for (int u = 0; u < kSrChains; u++) {
      const uint32_t j = j0 + u * groups;
      const double4 o = s_at[j];
      const bool same = kOwn && j == self;
      dx[u] = me.x - o.x;
      dy[u] = me.y - o.y;
      dz[u] = me.z - o.z;
      q[u] = same ? 0.0 : o.w;
      const double r2 = fma(dx[u], dx[u], fma(dy[u], dy[u], dz[u] * dz[u]));
      ir[u] = sr_rsqrt(same ? 1.0 : r2);
    }
#pragma unroll
    for (int u = 0; u < kSrChains; u++) {
      const double e = q[u] * ir[u];
      const double fs = e * (ir[u] * ir[u]);
      f[u].x = fma(fs, dx[u], f[u].x);
      f[u].y = fma(fs, dy[u], f[u].y);
      f[u].z = fma(fs, dz[u], f[u].z);
      f[u].e += e;
    }
  }
}

// A warp's share of a cell: chunks chunk0, chunk0 + warps_per_cell, ... of its
// atoms against row `row` of `rows`.
__device__ __forceinline__ void sr_warp(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
                                        const uint32_t *__restrict__ cell_point, const Grid &g, uint32_t natom,
                                        double4 *__restrict__ sr, uint32_t rows, uint32_t row, uint32_t cell,
                                        uint32_t chunk0, uint32_t warps_per_cell, uint32_t max_width,
                                        double4 *s_at) {
  const uint32_t cnt = cell_count[cell];
  const uint32_t width = min(max_width, cnt > 16 ? 32u : cnt > 8 ? 16u : 8u), groups = 32u / width;
  if (chunk0 * width >= cnt) return;
  const uint32_t lane = threadIdx.x & 31u, sub = lane / width, li = lane & (width - 1u);
  const uint32_t start = cell_point[cell];
  const int ix = cell / (g.ny * g.nz), iy = (cell / g.nz) % g.ny, iz = cell % g.nz;
  const uint32_t z0 = iz > 0 ? iz - 1 : 0, z1 = min(iz + 1, (int)g.nz - 1);
  const uint32_t n_runs = kSrRowsLines / rows;
  for (uint32_t a0 = chunk0 * width; a0 < cnt; a0 += warps_per_cell * width) {
    const bool active = a0 + li < cnt;
    const uint32_t i = start + a0 + li;
    const double4 me = active ? pd[i] : make_double4(0., 0., 0., 0.);
    const double4 none = make_double4(1e30, 1e30, 1e30, 0.);
    SrSum f4[kSrChains] = {};
    for (uint32_t q = 0; q < n_runs; q++) {
      const int t = row * n_runs + q, dx = t / 3 - 1, dy = t % 3 - 1;
      const int jx = ix + dx, jy = iy + dy;
      if (jx < 0 || jy < 0 || jx >= (int)g.nx || jy >= (int)g.ny) continue;
      const uint32_t c = (jx * g.ny + jy) * g.nz;
      uint32_t b = cell_point[c + z0];
      const uint32_t end = cell_point[c + z1] + cell_count[c + z1];
      const bool own = dx == 0 && dy == 0;
      double4 ahead = b + lane < end ? pd[b + lane] : none;
      for (; b < end; b += 32) {
        __syncwarp();
        s_at[lane] = ahead;
        __syncwarp();
        ahead = b + 32 + lane < end ? pd[b + 32 + lane] : none;
        const uint32_t n = min(32u, end - b);
        if (own) sr_batch<true>(s_at, n, sub, groups, me, i - b, f4);
        else sr_batch<false>(s_at, n, sub, groups, me, 0, f4);
      }
    }
    SrSum f;
    f.x = (f4[0].x + f4[1].x) + (f4[2].x + f4[3].x);
    f.y = (f4[0].y + f4[1].y) + (f4[2].y + f4[3].y);
    f.z = (f4[0].z + f4[1].z) + (f4[2].z + f4[3].z);
    f.e = (f4[0].e + f4[1].e) + (f4[2].e + f4[3].e);
    for (uint32_t o = width; o < 32; o <<= 1) {
      f.x += __shfl_xor_sync(0xffffffffu, f.x, o);
      f.y += __shfl_xor_sync(0xffffffffu, f.y, o);
      f.z += __shfl_xor_sync(0xffffffffu, f.z, o);
      f.e += __shfl_xor_sync(0xffffffffu, f.e, o);
    }
    if (active && sub == 0) {
      const double qi = me.w;
      sr[(size_t)row * natom + i] = make_double4(qi * f.x, qi * f.y, qi * f.z, qi * f.e);
    }
  }
}

// CTA: kSrWarps / warps_per_cell cells.
__device__ __forceinline__ void sr_block(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
                                         const uint32_t *__restrict__ cell_point, const Grid &g, uint32_t natom,
                                         double4 *__restrict__ sr, uint32_t rows, uint32_t warps_per_cell,
                                         uint32_t max_width, uint32_t bx, uint32_t row) {
  __shared__ double4 s_at[kSrWarps][32];
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t w = bx * kSrWarps + warp, cell = w / warps_per_cell;
  if (cell >= g.ncell) return;
  sr_warp(pd, cell_count, cell_point, g, natom, sr, rows, row, cell, w - cell * warps_per_cell, warps_per_cell,
          max_width, s_at[warp]);
}

__global__ void __launch_bounds__(kSrThreads)
k_short_range(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
              const uint32_t *__restrict__ cell_point, Grid g, uint32_t natom,
              double4 *__restrict__ sr, uint32_t rows, uint32_t warps_per_cell, uint32_t max_width) {
  sr_block(pd, cell_count, cell_point, g, natom, sr, rows, warps_per_cell, max_width, blockIdx.x, blockIdx.y);
}

// Lanes per chunk, at most: the widest chunks of which there are still 2,048
// (about four warps for each of the GPU's schedulers), else 8 atoms wide.
__host__ __device__ inline uint32_t sr_width(uint32_t natom, uint32_t rows) {
  const uint64_t lanes = (uint64_t)natom * rows;
  return lanes >= 2048u * 32u ? 32u : lanes >= 2048u * 16u ? 16u : 8u;
}

// Warps per cell for a mean number of atoms per cell.
__host__ __device__ inline uint32_t sr_warps_per_cell(uint32_t natom, uint32_t ncell, uint32_t width) {
  const uint32_t mean = natom / ncell;
  return 4 * mean <= 3 * width ? 1u : 4 * mean <= 7 * width ? 2u : 4u;
}

// ----------------------------------------------------------------------------
// Combine: near field + long-range partials (fixed order), write the
// cell-ordered outputs and scatter to input order; per-CTA energy sums.
// A CTA takes kCombineAtoms consecutive atoms; its warps split the partial
// rows (warp w sums rows w, w + 8, ... for the warp's 32 atoms, each load a
// coalesced 1 KB run), then warp 0 adds the eight row sums and the near-field
// planes in a fixed order.  (One thread per atom summing every row left small
// systems, with hundreds of rows and a few CTAs, latency-bound.)
constexpr int kCombineThreads = 256;
constexpr int kCombineAtoms = 32;
constexpr int kCombineWarps = kCombineThreads / 32;

// Total energy 0.5 * sum of the per-CTA sums, fixed order (one CTA).
__device__ __forceinline__ void energy_body(const double *block_energy, uint32_t nblocks,
                                            double *__restrict__ total) {
  __shared__ double s_red[32];
  double e = 0.0;
  for (uint32_t b = threadIdx.x; b < nblocks; b += blockDim.x) e += __ldcg(block_energy + b);
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (unsigned w = 0; w < (blockDim.x >> 5); w++) t += s_red[w];
    *total = 0.5 * t;
  }
}

__device__ __forceinline__ void combine_block(const double4 *__restrict__ sr, uint32_t sr_rows,
                                              const double4 *__restrict__ part,
                                              uint32_t nsplit, const uint32_t *__restrict__ sorted_idx,
                                              uint32_t natom, int use_far, double *__restrict__ cfx,
                                              double *__restrict__ cfy, double *__restrict__ cfz,
                                              double *__restrict__ cen, double *__restrict__ ofx,
                                              double *__restrict__ ofy, double *__restrict__ ofz,
                                              double *__restrict__ oen, double *__restrict__ block_energy,
                                              uint32_t nblocks, uint32_t *__restrict__ ticket,
                                              double *__restrict__ energy, uint32_t bx) {
  __shared__ double4 s_rows[kCombineWarps][kCombineAtoms];
  __shared__ bool s_last;
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t p = bx * kCombineAtoms + lane;
  const bool live = p < natom;
  double4 acc = make_double4(0., 0., 0., 0.);
  if (live && use_far) {
    for (uint32_t s = w; s < nsplit; s += kCombineWarps) {
      const double4 v = part[(size_t)s * natom + p];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
  }
  s_rows[w][lane] = acc;
  __syncthreads();
  double e = 0.0;
  if (w == 0 && live) {
    double4 t = s_rows[0][lane];
#pragma unroll
    for (int k = 1; k < kCombineWarps; k++) {
      const double4 v = s_rows[k][lane];
      t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    for (uint32_t pl = 0; pl < sr_rows; pl++) {
      const double4 v = sr[(size_t)pl * natom + p];
      t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    cfx[p] = t.x; cfy[p] = t.y; cfz[p] = t.z; cen[p] = t.w;
    const uint32_t i = sorted_idx[p];
    if (i < natom) { ofx[i] = t.x; ofy[i] = t.y; ofz[i] = t.z; oen[i] = t.w; }
    e = t.w;
  }
  if (w == 0) {
    for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if (lane == 0) {
      block_energy[bx] = e;
      // the CTA that draws the last ticket (they wrap to 0 by themselves)
      // sums the blocks' energies, in their order whichever CTA it is
      __threadfence();
      s_last = ticket && atomicInc(ticket, nblocks - 1) == nblocks - 1;
    }
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  energy_body(block_energy, nblocks, energy);
}

__global__ void __launch_bounds__(kCombineThreads)
k_combine(const double4 *__restrict__ sr, uint32_t sr_rows, const double4 *__restrict__ part, uint32_t nsplit,
          const uint32_t *__restrict__ sorted_idx, uint32_t natom, int use_far,
          double *__restrict__ cfx, double *__restrict__ cfy, double *__restrict__ cfz,
          double *__restrict__ cen, double *__restrict__ ofx, double *__restrict__ ofy,
          double *__restrict__ ofz, double *__restrict__ oen, double *__restrict__ block_energy,
          uint32_t *__restrict__ ticket, double *__restrict__ energy) {
  combine_block(sr, sr_rows, part, nsplit, sorted_idx, natom, use_far, cfx, cfy, cfz, cen, ofx, ofy, ofz, oen,
                block_energy, gridDim.x, ticket, energy, blockIdx.x);
}

// ----------------------------------------------------------------------------
// Sum of the per-atom outputs of the node-range shards of one system (the
// reference's reduce to GPU 0, src/glst_force.cu:1584-1602 with
// src/device_comm.cu:176-201 ncclReduce): dst[i] = src[0][i] + src[1][i] +
// ..., shards in order, for the four input-order and the four cell-order
// arrays.  The sources may live on other GPUs (read over NVLink through peer
// access).  Per-CTA energy sums as k_combine writes them.
constexpr int kMaxShards = 16;
struct ShardSet {
  const double *src[kMaxShards][8];  // per shard: ofx, ofy, ofz, oen, cfx, cfy, cfz, cen
  double *dst[8];
  uint32_t n;
};

__global__ void __launch_bounds__(kCombineThreads)
k_reduce_shards(ShardSet ss, uint32_t natom, double *__restrict__ block_energy) {
  __shared__ double s_red[kCombineThreads / 32];
  const uint32_t i = blockIdx.x * kCombineThreads + threadIdx.x;
  double e = 0.0;
  if (i < natom) {
#pragma unroll
    for (int a = 0; a < 8; a++) {
      double t = 0.0;
      for (uint32_t s = 0; s < ss.n; s++) t += ss.src[s][a][i];
      ss.dst[a][i] = t;
      if (a == 3) e = t;
    }
  }
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kCombineThreads / 32; w++) t += s_red[w];
    block_energy[blockIdx.x] = t;
  }
}

__global__ void k_energy_total(const double *__restrict__ block_energy, uint32_t nblocks,
                               double *__restrict__ total) {
  energy_body(block_energy, nblocks, total);
}

// ----------------------------------------------------------------------------
// Direct all-pairs Coulomb, FP64, open boundary (the reference's physics
// check, utils/coulomb.cu:14-82): thread per atom, the other atoms streamed
// through shared memory.
constexpr int kDirectThreads = 128;

__global__ void __launch_bounds__(kDirectThreads)
k_direct_coulomb(const double *__restrict__ rx, const double *__restrict__ ry, const double *__restrict__ rz,
                 const double *__restrict__ qc, uint32_t n, double *__restrict__ fx, double *__restrict__ fy,
                 double *__restrict__ fz, double *__restrict__ en) {
  __shared__ double4 s_at[kDirectThreads];
  const uint32_t i = blockIdx.x * kDirectThreads + threadIdx.x;
  const bool active = i < n;
  const double xi = active ? rx[i] : 0.0, yi = active ? ry[i] : 0.0, zi = active ? rz[i] : 0.0;
  const double qi = active ? qc[i] : 0.0;
  double f0 = 0.0, f1 = 0.0, f2 = 0.0, e0 = 0.0;
  for (uint32_t j0 = 0; j0 < n; j0 += kDirectThreads) {
    const uint32_t nj = min((uint32_t)kDirectThreads, n - j0);
    __syncthreads();
    if (threadIdx.x < nj) {
      const uint32_t j = j0 + threadIdx.x;
      s_at[threadIdx.x] = make_double4(rx[j], ry[j], rz[j], qc[j]);
    }
    __syncthreads();
    if (!active) continue;
    for (uint32_t k = 0; k < nj; k++) {
      if (j0 + k == i) continue;
      const double4 o = s_at[k];
      const double dx = xi - o.x, dy = yi - o.y, dz = zi - o.z;
      const double ir = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz)));
      const double e = qi * o.w * ir;
      const double fs = e * ir * ir;
      f0 = fma(fs, dx, f0);
      f1 = fma(fs, dy, f1);
      f2 = fma(fs, dz, f2);
      e0 += e;
    }
  }
  if (active) {
    fx[i] = f0;
    fy[i] = f1;
    fz[i] = f2;
    en[i] = e0;
  }
}

// ----------------------------------------------------------------------------
// Pipe-peak probes (roofline denominators).  Eight independent chains per
// thread keep the pipe busy; the results are stored so nothing is removed.
__global__ void k_probe_sfu(float *out, int iters) {
  float a[8];
#pragma unroll
  for (int u = 0; u < 8; u++) a[u] = 0.001f * (threadIdx.x + u);
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      float s, c;
      sfu_sincos(a[u], &s, &c);
      a[u] = s + c;  // 2 MUFU + 1 FADD
    }
  }
  float t = 0.f;
#pragma unroll
  for (int u = 0; u < 8; u++) t += a[u];
  out[blockIdx.x * blockDim.x + threadIdx.x] = t;
}

__global__ void k_probe_fma(float *out, int iters) {
  float a[8];
#pragma unroll
  for (int u = 0; u < 8; u++) a[u] = 0.001f * (threadIdx.x + u);
  const float m = 0.999f, b = 0.0001f;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 8; u++) a[u] = fmaf(a[u], m, b);
  }
  float t = 0.f;
#pragma unroll
  for (int u = 0; u < 8; u++) t += a[u];
  out[blockIdx.x * blockDim.x + threadIdx.x] = t;
}

}  // namespace dev
}  // namespace glst
