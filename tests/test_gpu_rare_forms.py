"""GPU parity of the far-field forms that plans of the shipped designs do not
reach: groups whose series would need more than the longest compiled one (every
atom by one sine and cosine per node), and more radial nodes per direction than
are staged at a time.

The library is built once more with lower limits (16 terms, 4 radial nodes), so
that an ordinary plan -- 7^3 cells at the default order: 36, 22 and 16 terms, 33,
27 and 19 radial nodes -- takes both forms, and a process of its own solves with
it, alone and in a work-list batch.  Bars as for the usual forms: the far field's
forces and per-atom energies to 1e-5 (an FP32 phase of up to 30 rad carries 2e-6
rad), one system's results bitwise the same in a batch.
"""
import importlib.util
import math
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from oracle import oracle, planner

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PKG = os.path.join(ROOT, "gauss-legendre-spherical-t_b200")
T0 = math.erfc(3.1) / 10.0
SOLVE = r"""
import sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import __graft_entry__
pkg = __graft_entry__.load_package()
pkg._lib = pkg.load_library(sys.argv[2])
pkg.set_tdesign_path(pkg.TDESIGN_STORE)
d = np.load(sys.argv[3])
n, tol, L, rcut = int(d["n"]), float(d["tol"]), float(d["L"]), float(d["rcut"])
atoms = [torch.tensor(d[k], device="cuda:0") for k in "xyzq"]
with pkg.GlstForce(n, tol, L, L, L, rcut=rcut) as f:
    f.calc_ener_force(*atoms)
    got = f.get_ef()
out = [torch.empty(n, dtype=torch.float64, device="cuda:0") for _ in range(4)]
with pkg.GlstBatch([dict(natom=n, tol=tol, box=(L, L, L), rcut=rcut)]) as b:
    b.compute(*atoms, *out, mode="worklist")
    torch.cuda.synchronize()
with open("/proc/self/maps") as m:
    assert sys.argv[2] in m.read()
np.savez(sys.argv[4], got=np.stack(got), batch=np.stack([o.cpu().numpy() for o in out]))
"""


@pytest.fixture(scope="module")
def small_limits(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("glst_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    lib = str(tmp_path_factory.mktemp("lib") / "libglst_small.so")
    return build.build(lib=lib, defines=["-DGLST_MAX_TERMS=16", "-DGLST_RAD_CHUNK=4"])


@pytest.mark.parametrize("n,L,rcut,tol", [(1501, 66.9, 10.0, T0), (300, 40.0, 10.0, 1e-4), (9000, 40.0, 10.0, 1e-3)])
def test_rare_forms_match_the_oracle(pkg, small_limits, store, tmp_path, n, L, rcut, tol):
    rng = np.random.default_rng(n)
    m = int(math.ceil(n ** (1 / 3)))
    lat = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    p = (lat + 0.5 + rng.uniform(-0.4, 0.4, lat.shape)) * L / m
    p[:20] -= 6.0  # outside the box, beyond the series' range
    p = p[rng.permutation(n)]
    x, y, z = (np.ascontiguousarray(p[:, i]) for i in range(3))
    q = rng.choice([-0.834, 0.417, 0.417], n)
    np.savez(tmp_path / "in.npz", x=x, y=y, z=z, q=q, n=n, tol=tol, L=L, rcut=rcut)
    subprocess.run([sys.executable, "-c", SOLVE, ROOT, small_limits, str(tmp_path / "in.npz"),
                    str(tmp_path / "out.npz")], check=True, timeout=300)
    out = np.load(tmp_path / "out.npz")
    plan = planner.make_plan(n, tol, (L, L, L), rcut, store)
    near, ref = oracle.glst(x, y, z, q, plan, far=False), oracle.glst(x, y, z, q, plan)

    def rms(a):
        return np.sqrt(np.mean(sum(v * v for v in a)))
    far = [r - s for r, s in zip(ref, near)]
    err = [g - r for g, r in zip(out["got"], ref)]
    assert rms(far[:3]) > 0.0
    assert rms(err[:3]) <= 1e-5 * rms(far[:3]) + 1e-12 * rms(ref[:3])
    assert rms(err[3:]) <= 1e-5 * rms(far[3:]) + 1e-12 * rms(ref[3:])
    assert np.array_equal(out["got"], out["batch"])
    # the usual library takes another route, to the same result
    with pkg.GlstForce(n, tol, L, L, L, rcut=rcut) as f:
        f.calc_ener_force(*[torch.tensor(v, device="cuda:0") for v in (x, y, z, q)])
        usual = np.stack(f.get_ef())
    assert not np.array_equal(out["got"], usual)
