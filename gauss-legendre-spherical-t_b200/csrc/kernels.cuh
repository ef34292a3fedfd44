// The far field's two passes over atoms, structure factors and gather (sm_100a):
// their arguments and device code.  far_field.cu compiles the kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "layout.cuh"

namespace glst {
namespace dev {

// ----------------------------------------------------------------------------
// Sine and cosine on the FP32 FMA pipe, for what the series below do not take:
// atoms beyond their range, and groups that would need too many terms.  Method:
// theta = n pi + r with n = rint(theta / pi) (rounded by adding 1.5 * 2^23),
// r = theta - n pi in two FMA steps (pi = kPiHi + kPiLo,
// kPiHi with 8 significant bits so n * kPiHi is exact), then
//   sin r = r + r^3 P(r^2),  cos r = Q(r^2)   on |r| <= pi/2,
// with P of degree 3 and Q of degree 4, coefficients fitted by this project
// (Lawson-weighted least squares on [0, (pi/2)^2], csrc/fit_sincos.py).
// sin(theta) = (-1)^n sin r, cos(theta) = (-1)^n cos r: the common sign is
// returned folded into a factor (the atom's charge) instead of applied to
// both results.  Max abs error 1.8e-7 for |theta| <= 30; n kPiHi is exact to
// |theta| = 2e5, where the phase itself is an FP32 number of 0.01 rad.  (Beyond
// 1e7 rad -- an atom 1e7 A outside the box -- the reduction fails.)
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
// 8 and 4 rad in water10k's groups): P = 36, 22 and 16 terms carry all 33,
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
// or not a number) take one sine and cosine per node instead.  So did tiles of
// up to P / 16 atoms, by a count of the issue slots; measured, the series wins
// from one atom on: 8^3 cells of 1 / 2 / 3 atoms at the default order 196 / 199 /
// 202 us against 265 / 353 / 403 (gather 230 / 230 / 230 against 448 / 632 / 767),
// 20^3 cells of one atom at 1e-3 103 against 128 (gather 135 against 133).
// Measured: water10k 1.112 -> 0.297 ms, 1,000 waters on 4^3 cells 0.144 ->
// 0.056 ms, 168 atoms per cell 0.313 -> 0.094 ms; forces 3.3e-8 -> 1.5e-8 off
// the FP64 path.
constexpr int kSfWarps = 4;
constexpr int kSfThreads = 32 * kSfWarps;
constexpr int kSfAtomTile = 128;
#ifndef GLST_RAD_CHUNK  // (smaller in a test's build, as GLST_MAX_TERMS)
#define GLST_RAD_CHUNK 64
#endif
#ifndef GLST_MAX_TERMS
#define GLST_MAX_TERMS 64
#endif
constexpr int kSfRadChunk = GLST_RAD_CHUNK;  // radial nodes staged at a time, at most
constexpr int kChebMaxP = GLST_MAX_TERMS;    // series terms, at most (the lengths compiled: planner, series_terms)
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

// Rows of the staged results are an odd number of float2 apart (bank spread).
__host__ __device__ constexpr uint32_t sf_row(uint32_t rc) { return rc | 1u; }

__host__ __device__ inline size_t sf_smem_bytes(uint32_t max_rad, uint32_t tab4) {
  const uint32_t rc = max_rad < (uint32_t)kSfRadChunk ? max_rad : (uint32_t)kSfRadChunk;
  return tab4 * sizeof(float4) + (size_t)kSfWarps * (32 * sizeof(float4) + 32 * sf_row(rc) * sizeof(float2));
}

// The general form, one sine and cosine per (atom, node), added to the staged
// results: the tile's atoms beyond the series' range (all: every atom).
static __device__ __noinline__ void sf_direct(const float4 *__restrict__ pk, uint32_t na, bool all, float u2, float4 s,
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
static __device__ __noinline__ void sf_store_dense(float2 f, size_t o, bool add, bool last, float2 *__restrict__ S,
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
    const bool series = P > 0 && na > 0;
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
// `cell0` on (cells far apart, which would spread a cluster's full cells, cost
// 2 % on 26^3 cells of 6 atoms and 6-10 % on a droplet and a slab there: S is
// written in longer runs this way).
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
#define GLST_SF_CASE(n)                                                                                           \
  case n:                                                                                                         \
    for (uint32_t cell = cell0; cell < cell1; cell++)                                                             \
      sf_tile<(n <= kChebMaxP ? n : 0)>(a, u, a.pk + a.cell_point[cell], a.cell_count[cell], cell, s_sf, s_at, s_f); \
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

// (blocks in x: quad fastest, then a.cells cells from cell_base on)
__global__ void k_structure_factors(const __grid_constant__ SfArgs a, uint32_t cell_base);

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
// tiles and warps.  Atoms beyond the series' range take a sine and cosine per
// node (lr_direct).
//
// Warps are independent: each takes a cell (up to its cap, then pieces of denser
// cells: layout.cuh) and a chunk of direction tiles, with no CTA barriers (four
// warps on one cell's chunk waited for each other a third of the time).  A tile's
// R' is copied to shared memory asynchronously while the previous tile's series
// are evaluated -- the buffer is free once its coefficients are formed.  The
// groups' tables are copied to shared memory where three CTAs per SM still fit
// with them (water10k 485 -> 478 us, 168 atoms per cell 149 -> 143, 648 atoms 47
// -> 42).  At 168 registers only the lengths above 48, which no shipped design
// reaches, spill.
// Measured: water10k 1.458 -> 0.485 ms, 3,000 atoms on 4^3 cells 0.141 ->
// 0.076 ms, 168 atoms per cell 0.279 -> 0.148 ms, a million atoms 55 -> 17 ms;
// forces 1.5e-8 -> 0.9e-8 off the FP64 path.
constexpr int kLrWarps = 4;
constexpr int kLrThreads = 32 * kLrWarps;
constexpr int kLrAtomTile = 128;
constexpr int kLrBatch = 8;       // atoms reduced across the warp together
// Refused by set-up, as ever (neither occurs for the shipped designs): more radial
// nodes per direction, more quads of radial nodes over all groups.
constexpr uint32_t kLrMaxRad = 256;
constexpr uint32_t kLrMaxQuads = 128;

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
  uint32_t n_chunks;
  Pieces pieces;
};

__host__ __device__ inline size_t lr_smem_bytes(uint32_t max_rad) {
  const uint32_t rc = max_rad < (uint32_t)kSfRadChunk ? max_rad : (uint32_t)kSfRadChunk;
  return (size_t)kLrWarps * (kLrAtomTile * (sizeof(float4) + 4 * sizeof(double)) + 32 * sf_row(rc) * sizeof(float2));
}

// The general form for a warp's 32 directions: the tile's atoms beyond the
// series' range (all: every atom), one sine and cosine per (atom, node).
static __device__ __noinline__ void lr_direct(const LrArgs &a, const DirTile &u, const float4 *__restrict__ atoms,
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

// Work item of a warp: the atoms [first, end) of a cell and a chunk of direction
// tiles.
template <bool kTabShared>
__device__ __forceinline__ void lr_warp(const LrArgs &a, uint32_t cell, uint32_t first, uint32_t end, uint32_t chunk) {
  extern __shared__ float4 s_lr[];
  const uint32_t cnt = min(a.cell_count[cell], end);
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t start = a.cell_point[cell];
  const uint32_t t0 = chunk * a.tiles_per_chunk, t1 = min(a.n_tiles, t0 + a.tiles_per_chunk);
  const uint32_t rc = min(a.max_rad, (uint32_t)kSfRadChunk);
  float4 *s_own = s_lr + (kTabShared ? a.tab4 : 0u);  // (the tables come first)
  float4 *s_at = s_own + warp * kLrAtomTile;
  double *acc = reinterpret_cast<double *>(s_own + kLrWarps * kLrAtomTile) + warp * (kLrAtomTile * 4);
  float2 *s_r = reinterpret_cast<float2 *>(reinterpret_cast<double *>(s_own + kLrWarps * kLrAtomTile) +
                                           kLrWarps * kLrAtomTile * 4) + (size_t)warp * 32 * sf_row(rc);
  for (uint32_t a0 = first; a0 < cnt; a0 += kLrAtomTile) {
    const uint32_t na = min((uint32_t)kLrAtomTile, cnt - a0), pad = (na + kLrBatch - 1) & ~(uint32_t)(kLrBatch - 1);
    // the first series tile
    auto is_series = [&](const DirTile &u) { return u.n_dir > 0 && u.lr_P > 0; };
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
  case n: lr_tile<(n <= kChebMaxP ? n : 4), kTabShared>(a, u, next, na, cell, s_at, acc, s_r); break;
      switch (u.lr_P) {
      GLST_LR_CASE(4) GLST_LR_CASE(6) GLST_LR_CASE(8) GLST_LR_CASE(10) GLST_LR_CASE(12)
      GLST_LR_CASE(14) GLST_LR_CASE(16) GLST_LR_CASE(18) GLST_LR_CASE(20) GLST_LR_CASE(22)
      GLST_LR_CASE(24) GLST_LR_CASE(26) GLST_LR_CASE(28) GLST_LR_CASE(30) GLST_LR_CASE(32)
      GLST_LR_CASE(34) GLST_LR_CASE(36) GLST_LR_CASE(40) GLST_LR_CASE(48) GLST_LR_CASE(56)
      GLST_LR_CASE(64)
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

// A warp's items: a cell (up to its cap) and a chunk, then pieces of dense cells
// with the same chunk.  Items chunk by chunk, so that the first (largest) groups'
// work starts first and a CTA's warps share a chunk's tables.
template <bool kTabShared>
__device__ __forceinline__ void lr_items(const LrArgs &a, uint32_t cell, uint32_t chunk) {
  uint32_t next = a.ncell - 1 - cell;
  const uint32_t n_pieces = next < kPieceWarps ? *a.pieces.n : 0u;
  for (uint32_t first = 0, end = a.pieces.cap;; next += min(a.ncell, kPieceWarps)) {
    lr_warp<kTabShared>(a, cell, first, end, chunk);
    if (next >= n_pieces) return;
    const uint2 r = a.pieces.list[next];
    cell = r.x;
    first = r.y;
    end = first + kPieceAtoms;
  }
}

// the general form reads the tables from global memory
__global__ void k_long_range(const __grid_constant__ LrArgs a);
__global__ void k_long_range_general(const __grid_constant__ LrArgs a);

// ----------------------------------------------------------------------------
// Many systems per launch (worklist.cuh).
struct SysDesc {
  Grid g;
  uint32_t natom, combine_blocks, part_rows, use_far, sr_rows;
  SatArgs sat;  // shell-sum arguments (S, node tables, nodes per CTA, row stride, R)
  const double *rx, *ry, *rz, *qc;
  uint32_t *atom_cell, *atom_slot, *perm, *sorted_idx, *cell_count, *cell_point;
  float4 *pk;
  double4 *pd;
  SfArgs sf;    // structure-factor arguments
  LrArgs lr;    // gather arguments
  double4 *part, *sr;
  uint32_t *ticket, *n_pieces;
  uint2 *piece_list;
  Pieces pieces;    // the same for its readers
  double *cfx, *cfy, *cfz, *cen, *ofx, *ofy, *ofz, *oen, *block_energy, *energy;
};

struct WorkItem {
  uint32_t sys, a, b, pad;
};

__global__ void k_structure_factors_multi(const SysDesc *__restrict__ sys, const WorkItem *__restrict__ items,
                                          uint32_t n);
__global__ void k_long_range_multi(const SysDesc *__restrict__ sys, const WorkItem *__restrict__ items, uint32_t n);

}  // namespace dev
}  // namespace glst
