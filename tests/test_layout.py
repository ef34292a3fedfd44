"""Host layout of the far field (CPU): tiles, stages, gather chunks and shards.

A small program built from planner.cpp prints far_layout's result; the checks
are its contract: the shards' nodes are contiguous, disjoint and complete, each
holds K / n nodes to within one tile (half a tile at either end), chunks cover
the stage's tiles, a quad never mixes groups.
"""
import math
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gauss-legendre-spherical-t_b200", "csrc")
T0 = math.erfc(3.1) / 10.0
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "planner.hpp"
int main(int argc, char **argv) {  // store natom tol bx by bz rcut waves stage_bytes nshards
  const double box[3] = {std::atof(argv[4]), std::atof(argv[5]), std::atof(argv[6])};
  auto store = glst::TDesignStore::open(argv[1]);
  const auto p = glst::make_plan(std::atoi(argv[2]), std::atof(argv[3]), box, std::atof(argv[7]), 0, *store);
  const unsigned n = std::atoi(argv[10]);
  std::printf("K %u\n", p.K());
  for (unsigned s = 0; s < n; s++) {
    const auto l = glst::far_layout(p, s, n, std::atoi(argv[8]), 148, std::strtoull(argv[9], nullptr, 10));
    std::printf("shard %u %u %u %u\n", l.k_begin, l.K, l.stage_kmax, l.part_rows);
    for (const auto &t : l.tiles) std::printf("tile %u %u %u %u\n", t.group, t.n_dir, t.kb, t.ke);
    for (const auto &g : l.stages) std::printf("stage %u %u %u %u %u\n", g.kb, g.ke, g.u0, g.u1, g.tpc);
  }
}
"""


@pytest.fixture(scope="module")
def layout(tmp_path_factory, pkg):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("layout")
    with open(d / "main.cpp", "w") as f:
        f.write(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-o", str(d / "main"),
                    str(d / "main.cpp"), os.path.join(CSRC, "planner.cpp")], check=True)

    def run(natom, tol, box, rcut, waves=4, stage_bytes=4 << 30, nshards=1):
        out = subprocess.run([str(d / "main"), pkg.TDESIGN_STORE, str(natom), repr(tol), *map(repr, box), repr(rcut),
                              str(waves), str(stage_bytes), str(nshards)], check=True, capture_output=True, text=True)
        K, shards = 0, []
        for line in out.stdout.split("\n"):
            w = line.split()
            v = [int(a) for a in w[1:]]
            if not w:
                continue
            if w[0] == "K":
                K = v[0]
            elif w[0] == "shard":
                shards.append(dict(k=v[0], K=v[1], kmax=v[2], rows=v[3], tiles=[], stages=[]))
            else:
                shards[-1][w[0] + "s"].append(v)
        return K, shards
    return run


CASES = [(30000, T0, (66.9,) * 3, 10.0), (100000, 1e-3, (260.0,) * 3, 10.0), (6000, 1e-5, (39.1,) * 3, 10.0),
         (30000, 0.1 * T0, (66.9,) * 3, 10.0), (12000, T0, (41.5, 58.3, 39.1), 10.0)]


@pytest.mark.parametrize("nshards", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("natom,tol,box,rcut", CASES)
def test_shards_are_even(layout, natom, tol, box, rcut, nshards):
    K, shards = layout(natom, tol, box, rcut, nshards=nshards)
    biggest = max(t[3] - t[2] for s in shards for t in s["tiles"])
    assert sum(s["K"] for s in shards) == K
    at = 0
    for s in shards:
        if s["K"]:
            assert s["k"] == at
        at += s["K"]
        assert abs(s["K"] - K / nshards) <= biggest + 1


@pytest.mark.parametrize("stage_bytes", [1 << 20, 16 << 20, 4 << 30])
@pytest.mark.parametrize("natom,tol,box,rcut", CASES)
def test_stages_and_chunks_cover_the_tiles(layout, natom, tol, box, rcut, stage_bytes):
    for waves, nshards in ((4, 1), (32, 1), (2, 3)):
        K, shards = layout(natom, tol, box, rcut, waves=waves, stage_bytes=stage_bytes, nshards=nshards)
        for s in shards:
            at = k = 0
            for kb, ke, u0, u1, tpc in s["stages"]:
                assert u0 == at and (u1 - u0) % 4 == 0 and kb == k and tpc >= 1
                tiles = s["tiles"][u0:u1]
                for i in range(0, len(tiles), 4):
                    assert len({t[0] for t in tiles[i:i + 4]}) == 1  # one group per quad
                real = [t for t in tiles if t[1]]
                assert real[0][2] - s["k"] == kb and real[-1][3] - s["k"] == ke
                assert all(a[3] == b[2] for a, b in zip(real, real[1:]))
                assert all(1 <= t[1] <= 32 for t in real)
                assert -(-(u1 - u0) // tpc) <= s["rows"] and ke - kb <= s["kmax"]
                at, k = u1, ke
            assert at == len(s["tiles"]) and k == s["K"]
