"""How the work over cells is divided (CPU): the rules of layout.cuh.

Several cells share a structure-factor CTA only where cells hold few atoms and
enough CTAs are left to fill the GPU: at least 12 per SM at eight cells each.
"""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gauss-legendre-spherical-t_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include "layout.cuh"
using namespace glst::dev;
int main() {
  unsigned natom, ncell, quads;
  while (std::scanf("%u %u %u", &natom, &ncell, &quads) == 3) std::printf("%u\n", sf_cells(natom, ncell, quads));
}
"""


@pytest.fixture(scope="module")
def sf_cells(tmp_path_factory):
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
        return [int(v) for v in out.stdout.split()]
    return run


def test_cells_per_structure_factor_cta(sf_cells):
    args = [(n, c ** 3, q) for c in (1, 3, 4, 6, 8, 11, 16, 22, 26, 60) for q in (1, 5, 15, 32, 200)
            for n in (1, 417, 2 * c ** 3, 16 * c ** 3, 17 * c ** 3, 100 * c ** 3)]
    for (n, c, q), cells in zip(args, sf_cells(args)):
        assert cells in (1, 4, 8)
        if cells > 1:
            assert n // c <= 16 and c * q // 8 >= 12 * 148
    # 139 waters at an 8 A cutoff; 33,333 waters on 26^3 cells
    assert sf_cells([(417, 27, 15), (99999, 17576, 5)]) == [1, 8]
