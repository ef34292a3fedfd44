// Cell assignment, near field, combine and reductions, the direct-sum check and
// the pipe-peak probes (sm_100a).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "layout.cuh"

namespace glst {
namespace dev {

constexpr unsigned kSortCap = 8192;   // atoms per cell the shared-memory cell sort holds

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
// consecutive cells per thread and step: 26^3 cells in 5 steps instead of 18),
// and the pieces of cells of more than `cap` atoms (layout.cuh; pieces may be null).
// The pieces' order varies, what is computed of a piece does not depend on it.
__device__ __forceinline__ void scan_body(const uint32_t *__restrict__ cell_count, uint32_t ncell,
                                          uint32_t *__restrict__ cell_point, uint32_t cap, uint2 *__restrict__ pieces,
                                          uint32_t *__restrict__ n_pieces) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t s_pieces;
  if (threadIdx.x == 0) s_pieces = 0;
  __syncthreads();
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
      if (pieces && v[u] > cap) {
        const uint32_t n = (v[u] - cap + kPieceAtoms - 1) / kPieceAtoms, at = atomicAdd(&s_pieces, n);
        for (uint32_t t = 0; t < n; t++) pieces[at + t] = make_uint2(c + u, cap + t * kPieceAtoms);
      }
    }
    __syncthreads();  // warp_sums is rewritten
  }
  if (pieces && threadIdx.x == 0) *n_pieces = s_pieces;
}

__global__ void k_scan(const uint32_t *__restrict__ cell_count, uint32_t ncell,
                       uint32_t *__restrict__ cell_point, uint32_t cap, uint2 *__restrict__ pieces,
                       uint32_t *__restrict__ n_pieces) {
  scan_body(cell_count, ncell, cell_point, cap, pieces, n_pieces);
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
// indices, then the whole CTA for each larger one.  A CTA's cells are far apart
// in the grid, so that a cluster's full cells, which lie together, go to
// different CTAs.  Launched with 32 kSortCells threads and kSortCap u32 of
// dynamic shared memory.
// Measured, a warp per cell against a CTA per cell: 26^3 cells of 12 / 28 / 60 /
// 87 atoms 16 / 30 / 67 / 130 us against 67 / 82 / 128 / 192; 7^3 cells 11 / 11 /
// 13 / 15 against 11 / 13 / 14 / 14.  (Up to 32 atoms only, the rest by the CTA:
// 7^3 cells of 28 atoms 24, of 40 atoms 40.)
constexpr uint32_t kSortWarpCap = 128;
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
  const uint32_t stride = (g.ncell + kSortCells - 1) / kSortCells, cell = bx + warp * stride;
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
    const uint32_t c = bx + w * stride;
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
// water10k 0.291 -> 0.187 ms, 168 atoms per cell 0.400 -> 0.258 ms, 26^3 cells
// of 6 atoms 0.485 -> 0.102 ms, 3,000 atoms on 4^3 cells 0.067 -> 0.045 ms, a
// million atoms 4.44 -> 4.25 ms.
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

// A warp's share of a cell: its atoms first, first + step, ... (`width` of them
// each time) below `end` against row `row` of `rows`.
__device__ __forceinline__ void sr_warp(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
                                        const uint32_t *__restrict__ cell_point, const Grid &g, uint32_t natom,
                                        double4 *__restrict__ sr, uint32_t rows, uint32_t row, uint32_t cell,
                                        uint32_t first, uint32_t step, uint32_t end, uint32_t width,
                                        double4 *s_at) {
  const uint32_t groups = 32u / width;
  const uint32_t lane = threadIdx.x & 31u, sub = lane / width, li = lane & (width - 1u);
  const uint32_t start = cell_point[cell];
  const int ix = cell / (g.ny * g.nz), iy = (cell / g.nz) % g.ny, iz = cell % g.nz;
  const uint32_t z0 = iz > 0 ? iz - 1 : 0, z1 = min(iz + 1, (int)g.nz - 1);
  const uint32_t n_runs = kSrRowsLines / rows;
  for (uint32_t a0 = first; a0 < end; a0 += step) {
    const bool active = a0 + li < end;
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
      const uint32_t e = cell_point[c + z1] + cell_count[c + z1];
      const bool own = dx == 0 && dy == 0;
      double4 ahead = b + lane < e ? pd[b + lane] : none;
      for (; b < e; b += 32) {
        __syncwarp();
        s_at[lane] = ahead;
        __syncwarp();
        ahead = b + 32 + lane < e ? pd[b + 32 + lane] : none;
        const uint32_t n = min(32u, e - b);
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

// Pieces next, next + step, ... of dense cells, `max_width` atoms at a time.  Out
// of line: in one loop with the cells' own atoms both were 5-6 % slower.
template <int kCtas>
static __device__ __noinline__ void sr_pieces(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
                                             const uint32_t *__restrict__ cell_point, const Grid &g, uint32_t natom,
                                             double4 *__restrict__ sr, uint32_t rows, uint32_t row, uint32_t max_width,
                                             const Pieces &pieces, uint32_t next, uint32_t step, double4 *s_at) {
  const uint32_t per = kPieceAtoms / max_width, n_pieces = *pieces.n * per;
  for (; next < n_pieces; next += step) {
    const uint2 r = pieces.list[next / per];
    const uint32_t first = r.y + (next % per) * max_width, end = min(cell_count[r.x], first + max_width);
    if (first < end)
      sr_warp(pd, cell_count, cell_point, g, natom, sr, rows, row, r.x, first, kPieceAtoms, end, max_width, s_at);
  }
}

// CTA: kSrWarps / warps_per_cell cells, up to pieces.cap atoms of each; then its
// warps take pieces of dense cells.
template <int kCtas>
__device__ __forceinline__ void sr_block(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
                                         const uint32_t *__restrict__ cell_point, const Grid &g, uint32_t natom,
                                         double4 *__restrict__ sr, uint32_t rows, uint32_t warps_per_cell,
                                         uint32_t max_width, const Pieces &pieces, uint32_t bx, uint32_t row) {
  __shared__ double4 s_at[kSrWarps][32];
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t w = bx * kSrWarps + warp, warps = g.ncell * warps_per_cell;
  const uint32_t cell = w / warps_per_cell;
  if (cell >= g.ncell) return;
  const uint32_t cnt = cell_count[cell];
  const uint32_t width = min(max_width, cnt > 16 ? 32u : cnt > 8 ? 16u : 8u);
  const uint32_t first = (w - cell * warps_per_cell) * width, end = min(cnt, pieces.cap);
  const uint32_t back = warps - 1 - w;
  const bool more = back < kPieceWarps && pieces.list && back < *pieces.n * (kPieceAtoms / max_width);
  if (first < end)
    sr_warp(pd, cell_count, cell_point, g, natom, sr, rows, row, cell, first, warps_per_cell * width, end, width,
            s_at[warp]);
  if (more)
    sr_pieces<kCtas>(pd, cell_count, cell_point, g, natom, sr, rows, row, max_width, pieces, back,
                     min(warps, kPieceWarps), s_at[warp]);
}

// kCtas: CTAs per SM the registers are cut for (sr_ctas).
template <int kCtas>
__global__ void __launch_bounds__(kSrThreads, kCtas)
k_short_range(const double4 *__restrict__ pd, const uint32_t *__restrict__ cell_count,
              const uint32_t *__restrict__ cell_point, Grid g, uint32_t natom,
              double4 *__restrict__ sr, uint32_t rows, uint32_t warps_per_cell, uint32_t max_width, Pieces pieces) {
  sr_block<kCtas>(pd, cell_count, cell_point, g, natom, sr, rows, warps_per_cell, max_width, pieces, blockIdx.x,
                  blockIdx.y);
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
// SFU sine and cosine of an FP32 angle in radians (PTX sin/cos.approx,
// flush-to-zero).
__device__ __forceinline__ void sfu_sincos(float x, float *s, float *c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}

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
