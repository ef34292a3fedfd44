// Host-side planning for one GLST system: cell grid, alpha groups and the
// cubature node set.  All FP64, as the reference's host code; see planner.cpp
// for the reference file:line each step follows.
#pragma once

#include <cstdint>
#include <map>
#include <mutex>
#include <memory>
#include <string>
#include <vector>

namespace glst {

struct PlanError {
  int status;  // glst_status
  std::string msg;
};

// Antipodal spherical t-designs keyed by degree; only the free half (m unit
// vectors) is kept, the full design being {p} U {-p}.
class TDesignStore {
 public:
  // `path`: a binary store (magic GLSTTD01) or a directory in the
  // reference's layout (files ssTTT.NNNNN).
  static std::shared_ptr<TDesignStore> open(const std::string &path);
  // Returns nullptr when the degree is not available.
  const std::vector<double> *get(unsigned t);  // 3*m doubles, xyz interleaved
  const std::string &path() const { return path_; }

 private:
  std::string path_;
  bool is_dir_ = false;
  std::map<unsigned, std::string> files_;  // degree -> file (dir layout)
  std::map<unsigned, unsigned> file_m_;    // degree -> N/2 (dir layout)
  std::map<unsigned, std::vector<double>> cache_;  // node-based: pointers stay valid
  std::mutex mu_;  // get() fills cache_ lazily (directory layout) from any thread
};

struct GroupPlan {
  unsigned width = 0;
  double rmax = 0, alpha = 0, zcut = 0;
  unsigned r_in = 0, r_out = 0;
  unsigned gl_degree = 0, t_degree = 0;
  unsigned n_radial = 0, n_dir = 0;
  std::vector<double> kappa;  // radial scales 2 alpha zcut x_i (n_radial)
  std::vector<double> dirs;   // unit directions s_j, xyz interleaved (3 n_dir)
  // Chebyshev series of the phases (below): terms, and n_radial rows of
  // series_row(P) floats -- of the structure factors (product basis) and of the
  // gather (plain)
  unsigned sf_P = 0, lr_P = 0;
  std::vector<float> sf_tab, lr_tab;
};

// Terms, at most (a test builds the library with less, to reach the kernels'
// forms for plans that the shipped designs do not give).
#ifndef GLST_MAX_TERMS
#define GLST_MAX_TERMS 64
#endif
constexpr unsigned kSeriesMaxP = GLST_MAX_TERMS;
constexpr unsigned series_b(unsigned P) { return P > 24 ? 8 : 4; }              // basis T_{Bg} T_b
constexpr unsigned series_row(unsigned P) { return (P + 3) / 4 * 4; }

struct Plan {
  uint32_t natom = 0;
  double tol = 0;
  double box[3] = {0, 0, 0};
  int ct_float = 0;
  uint32_t n[3] = {0, 0, 0};
  uint32_t ncell = 0;
  double cell_dim = 0;  // CT value widened to double
  // 1 / U in FP32, U the series' range: the radius of the cell's circumscribed
  // sphere and 2 % (atoms slightly outside the box stay within).  Coordinates
  // are scaled by it in FP32, so U is the reciprocal of an FP32 number: a
  // rounded scale would stretch every phase alike.
  float inv_u = 0;
  bool has_far = false;
  std::vector<GroupPlan> groups;
  // Node set in the reference's order, FP64 (pre-CT-rounding).
  std::vector<double> kx, ky, kz, w;
  std::vector<uint32_t> group;
  uint32_t K() const { return static_cast<uint32_t>(kx.size()); }
};

// Throws PlanError.
Plan make_plan(uint32_t natom, double tol, const double box[3], double rcut,
               int ct_float, TDesignStore &store);
double rcut_from_ncell(const double box[3], const uint32_t ncell[3]);

// How a handle works through its nodes (internal order: group -> direction ->
// radial).  They are cut into tiles of up to kTileDirs directions of one
// group, one warp each of the structure factors and the gather.  A shard of a
// system split over several devices takes a contiguous run of tiles (the
// reference splits its node list into contiguous per-GPU ranges,
// src/glst_force.cu:276-293).  Its tiles are run in stages of about equal node
// count, as many as keep S + R within the stage budget, and a stage's in gather
// chunks of tpc tiles, each with a partial row of 32 bytes per atom.  A group's
// tiles in a stage are padded to whole quads (a structure-factor CTA's warps
// share one group's table).  FP32 sums stay within a tile, everything across
// tiles is FP64, so neither shards nor stages nor chunks change a result beyond
// FP64 rounding.
constexpr unsigned kTileDirs = 32, kTileQuad = 4, kNodePad = 32;  // nodes of S and R are padded to kNodePad

struct FarLayout {
  struct Tile {
    uint32_t group, dir, n_dir;  // group, first direction within it, directions (0: padding)
    uint32_t kb, ke;             // nodes of the system
  };
  struct Stage {
    uint32_t kb, ke;             // nodes of the stage, from k_begin on
    uint32_t u0, u1;             // its tiles
    uint32_t tpc;                // tiles per gather chunk
    uint32_t rows() const { return (u1 - u0 + tpc - 1) / tpc; }  // gather chunks
  };
  std::vector<Tile> tiles;
  std::vector<Stage> stages;
  uint32_t k_begin = 0, K = 0;   // the shard's nodes
  uint32_t stage_kmax = 0;       // nodes of the largest stage
  uint32_t part_rows = 1;        // gather chunks of the largest stage
};

// `waves`: waves of gather warps to cut a stage's chunks for; `nsm`: SMs;
// `stage_bytes`: of S + R.
FarLayout far_layout(const Plan &p, uint32_t shard, uint32_t nshards, uint32_t waves, int nsm, uint64_t stage_bytes);

// Chebyshev (Jacobi-Anger) series of the phases of one direction,
//   e^{-i z x} = sum_p c_p(z) i^{p mod 2} T_p(x),  |x| <= 1,
// even p giving the real and odd p the imaginary part.
// series_terms: number of terms (even; above 48, with weights above 36, in
// larger steps; 0 when more than max_terms would be needed).  Without weights
// every z of the list is exact to below the rounding of an FP32 phase; with the
// weights w of a sum over the list, the sum and its derivative are.
// phase_series: the signed coefficients; product_basis: their conversion to
// the basis T_{Bg} T_b, p = Bg + b, b < B (in place).
unsigned series_terms(const std::vector<double> &z, const double *w, unsigned max_terms);
void phase_series(double z, unsigned P, double *c);
void product_basis(unsigned P, unsigned B, double *c);

// Exposed for tests of the numerics set-up.
double erfc_inverse(double y, double tol);
std::vector<double> gauss_legendre_roots(unsigned n);

}  // namespace glst
