"""The phases' Chebyshev series (CPU): planner.cpp's three functions.

A small program built from planner.cpp prints the number of terms for a list of
phases z and the coefficients; the series is summed here in FP64 and compared
with e^{-i z x} on |x| <= 1 -- plainly, and in the product basis T_{Bg} T_b that
the kernels use.  Bounds: what the number of terms leaves out (2e-7 of the
largest phase of a list, a weighted mean of 1e-8 with weights), and 1e-13 of
rounding where terms are ample.
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
#include <cstring>
#include "planner.hpp"
int main(int, char **argv) {
  unsigned P, n;
  double z;
  if (!std::strcmp(argv[1], "terms")) {  // weights? n z [w] ...
    unsigned weights;
    while (std::scanf("%u %u", &weights, &n) == 2) {
      std::vector<double> zs(n), ws(n);
      for (unsigned i = 0; i < n; i++) std::scanf(weights ? "%lf %lf" : "%lf", &zs[i], &ws[i]);
      std::printf("%u\n", glst::series_terms(zs, weights ? ws.data() : nullptr, glst::kSeriesMaxP));
    }
  } else {  // P z
    while (std::scanf("%u %lf", &P, &z) == 2) {
      std::vector<double> c(P), b(P);
      glst::phase_series(z, P, c.data());
      b = c;
      glst::product_basis(P, glst::series_b(P), b.data());
      for (unsigned p = 0; p < P; p++) std::printf("%.17g %.17g ", c[p], b[p]);
      std::printf("%u\n", glst::series_b(P));
    }
  }
}
"""


@pytest.fixture(scope="module")
def planner_fn(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("series")
    with open(d / "main.cpp", "w") as f:
        f.write(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-o", str(d / "main"),
                    str(d / "main.cpp"), os.path.join(CSRC, "planner.cpp")], check=True, capture_output=True)

    def run(what, text):
        out = subprocess.run([str(d / "main"), what], input=text, check=True, capture_output=True, text=True)
        return [[float(v) for v in line.split()] for line in out.stdout.splitlines()]
    return run


X = np.cos(np.linspace(0.0, np.pi, 401))


def _series(coef, basis):
    """sum_p coef_p i^{p mod 2} basis_p(X)."""
    s = np.zeros(X.size, dtype=complex)
    for p, c in enumerate(coef):
        s += c * (1j if p % 2 else 1.0) * basis(p)
    return s


def _error(row, z):
    """Largest |series - e^{-izx}|: plain and in the product basis."""
    B, c = int(row[-1]), np.array(row[:-1]).reshape(-1, 2)

    def T(p):
        return np.cos(p * np.arccos(X))
    exact = np.exp(-1j * z * X)
    return (np.max(np.abs(_series(c[:, 0], T) - exact)),
            np.max(np.abs(_series(c[:, 1], lambda p: T(p // B * B) * T(p % B)) - exact)))


def test_series_reconstruct_the_phase(planner_fn):
    # ample terms: rounding only; P as long as the kernels are compiled for
    cases = [(P, z) for P in (4, 6, 8, 16, 24, 26, 36, 48, 52, 64) for z in (0.0, 1e-9, 1e-3, 0.3, 1.0, 4.0, 11.0, 25.0)
             if P >= 1.35 * z + 14 or (P >= 8 and z <= 1e-3) or z <= 1e-9]
    assert len({P for P, _ in cases}) == 10
    rows = planner_fn("coef", "\n".join("%d %.17g" % c for c in cases))
    for (P, z), row in zip(cases, rows):
        plain, product = _error(row, z)
        # the product basis adds up to P / B coefficients of magnitude <= 2
        assert plain <= 1e-13 + z ** P and product <= 4e-13 + z ** P, (P, z, plain, product)


def test_number_of_terms_bounds_what_is_left_out(planner_fn):
    zs = [0.0, 1e-6, 0.01, 0.3, 1.0, 2.5, 4.0, 8.0, 12.0, 18.0, 25.0, 32.0, 40.0, 45.0]
    terms = [int(r[0]) for r in planner_fn("terms", "\n".join("0 1 %.17g" % z for z in zs))]
    lengths = set(range(4, 49, 2)) | {52, 56, 60, 64}
    for z, P in zip(zs, terms):
        assert P in lengths or (P == 0 and z > 40.0), (z, P)
    assert terms == sorted(t for t in terms if t) + [0] * terms.count(0)
    known = [(P, z) for P, z in zip(terms, zs) if P]
    for (P, z), row in zip(known, planner_fn("coef", "\n".join("%d %.17g" % c for c in known))):
        plain, product = _error(row, z)
        assert plain <= 2.1e-7 and product <= 2.1e-7, (P, z, plain, product)
    # a list takes what its largest phase takes
    a, b = planner_fn("terms", "0 4 0.1 3 18 7\n0 1 18")
    assert a == b


def test_number_of_terms_with_weights(planner_fn):
    # a Gaussian rule like the cubature's: the weighted mean of what is left out
    x = (np.arange(30) + 0.5) / 30
    for zmax, zc in ((18.0, 3.0), (8.0, 2.5), (30.0, 4.0), (40.0, 1.0)):
        z, w = zmax * x, np.exp(-(zc * x) ** 2)
        text = "1 30 " + " ".join("%.17g %.17g" % p for p in zip(z, w))
        P = int(planner_fn("terms", text)[0][0])
        assert P in set(range(4, 37, 2)) | {40, 48, 56, 64}, P
        rows = planner_fn("coef", "\n".join("%d %.17g" % (P, v) for v in z))
        left = sum(wi * zi * _error(row, zi)[0] for wi, zi, row in zip(w, z, rows)) / np.sum(w * z)
        assert left <= 1.1e-8, (zmax, P, left)
    # more than the longest series: none
    assert planner_fn("terms", "1 1 60 1")[0] == [0]
