// Shell sums of the structure factors over the cell grid (sm_100a).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "layout.cuh"

namespace glst {
namespace dev {

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

}  // namespace dev
}  // namespace glst
