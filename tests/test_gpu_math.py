"""The near field's reciprocal square root (two Newton steps from the
hardware's approximation) against long double and CUDA's rsqrt.

Bound: 1.5 x 2^-53 of rounding (the residual's product and the result) and
1e-17 of the iteration; the approximation has to be within 2^-15 for that.
Zero, infinity and not-a-number are CUDA's; a square below the smallest normal
number counts as zero.
"""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

CSRC = os.path.join(ROOT, "gauss-legendre-spherical-t_b200", "csrc")
SOURCE = r"""
#include <cstdio>
#include <vector>
#include "cells.cuh"
__global__ void k(const double *x, double *own, double *lib, unsigned n) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  own[i] = glst::dev::sr_rsqrt(x[i]);
  lib[i] = rsqrt(x[i]);
}
int main(int, char **argv) {
  std::vector<double> x(1 << 20), y(2 << 20);
  FILE *f = std::fopen(argv[1], "rb");
  const unsigned n = (unsigned)std::fread(x.data(), 8, x.size(), f);
  std::fclose(f);
  double *d;
  if (cudaMalloc(&d, 3ull * n * 8) != cudaSuccess) return 1;
  cudaMemcpy(d, x.data(), n * 8ull, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2ull * n, n);
  if (cudaMemcpy(y.data(), d + n, 2ull * n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  f = std::fopen(argv[2], "wb");
  std::fwrite(y.data(), 8, 2ull * n, f);
  std::fclose(f);
  return 0;
}
"""


def test_near_field_rsqrt(tmp_path):
    src, exe = str(tmp_path / "rsqrt.cu"), str(tmp_path / "rsqrt")
    with open(src, "w") as f:
        f.write(SOURCE)
    nvcc = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else "nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + CSRC,
                    "-o", exe, src], check=True, capture_output=True)
    rng = np.random.default_rng(11)
    tiny = np.finfo(np.float64).tiny
    # every exponent of a normal number (mantissas at random and at the ends),
    # and a dense sweep of two octaves
    e = np.arange(-1022, 1024)
    m = np.concatenate([1.0 + rng.random((200, e.size)), np.ones((1, e.size)), np.full((1, e.size), 2.0 - 2.0**-52)])
    x = np.concatenate([np.ldexp(m, e[None, :]).ravel(), np.linspace(1.0, 4.0, 400001)])
    special = np.array([0.0, np.inf, np.nan, tiny, np.finfo(np.float64).max, 5e-324, tiny / 2])
    allx = np.concatenate([x, special])
    assert allx.size <= 1 << 20
    allx.tofile(str(tmp_path / "x"))
    subprocess.run([exe, str(tmp_path / "x"), str(tmp_path / "y")], check=True)
    own, lib = np.fromfile(str(tmp_path / "y")).reshape(2, -1)
    true = 1.0 / np.sqrt(x.astype(np.longdouble))
    err = np.max(np.abs((own[:x.size] - true) / true))
    assert err <= 1.5 * 2.0**-53 + 1e-17, float(err)
    # ... so never more than two units in the last place from CUDA's (1 ulp)
    assert np.max(np.abs(own[:x.size] - lib[:x.size]) / np.spacing(lib[:x.size])) <= 2.0
    s, ls = own[x.size:], lib[x.size:]
    assert s[0] == ls[0] == np.inf and s[1] == ls[1] == 0.0 and np.isnan(s[2]) and np.isnan(ls[2])
    assert np.all(np.abs(s[3:5] / ls[3:5] - 1.0) < 1e-15)
    assert s[5] == s[6] == np.inf
