"""How the work over cells is divided (CPU): the rules of layout.cuh.

Several cells share a structure-factor CTA only where cells hold few atoms and
enough CTAs are left to fill the GPU: at least 12 per SM at eight cells each.
The list of dense cells' pieces holds whatever the atoms' distribution makes.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gauss-legendre-spherical-t_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "layout.cuh"
using namespace glst::dev;
int main() {
  unsigned natom, ncell, quads;
  while (std::scanf("%u %u %u", &natom, &ncell, &quads) == 3)
    std::printf("%u %u %u\n", sf_cells(natom, ncell, quads), cell_cap(natom, ncell), max_pieces(natom, ncell));
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    gxx, cuda = shutil.which("g++"), "/usr/local/cuda/include"
    if not gxx or not os.path.isdir(cuda):
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("division")
    with open(d / "main.cpp", "w") as f:
        f.write(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I" + CSRC, "-I" + cuda, "-o", str(d / "main"), str(d / "main.cpp")],
                   check=True)

    def run(args):
        out = subprocess.run([str(d / "main")], input="\n".join("%d %d %d" % a for a in args), check=True,
                             capture_output=True, text=True)
        return [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]
    return run


def test_cells_per_structure_factor_cta(rules):
    args = [(n, c ** 3, q) for c in (1, 3, 4, 6, 8, 11, 16, 22, 26, 60) for q in (1, 5, 15, 32, 200)
            for n in (1, 417, 2 * c ** 3, 16 * c ** 3, 17 * c ** 3, 100 * c ** 3)]
    for (n, c, q), (cells, _cap, _pieces) in zip(args, rules(args)):
        assert cells in (1, 4, 8)
        if cells > 1:
            assert n // c <= 16 and c * q // 8 >= 12 * 148
    # 139 waters at an 8 A cutoff; 33,333 waters on 26^3 cells
    assert [r[0] for r in rules([(417, 27, 15), (99999, 17576, 5)])] == [1, 8]


def test_pieces_of_dense_cells_fit_the_list(rules):
    rng = np.random.default_rng(2)
    counts = []
    for ncell in (1, 27, 343, 1000):
        for n in (1, 31, 32, 33, 64, 65, 1000, 30011):
            for p in (np.ones(ncell), rng.random(ncell) ** 20, np.arange(ncell) < 1, np.arange(ncell) < 2):
                counts.append(rng.multinomial(n, p / p.sum()))
            if n > ncell:  # one atom too many in as many cells as there are atoms for
                cap = rules([(n, ncell, 1)])[0][1]
                full = min(ncell, n // (cap + 1))
                counts.append(np.array([cap + 1] * full + [0] * (ncell - full)))
    for cnt, (_c, cap, pieces) in zip(counts, rules([(int(c.sum()), len(c), 1) for c in counts])):
        assert cap >= 32 and cap % 32 == 0 and cap >= cnt.sum() // len(cnt)
        assert np.sum((np.maximum(cnt - cap, 0) + 31) // 32) <= pieces
