"""GPU parity of the far field's Chebyshev series and of the near field's lane
groups at the sizes where they change form, against the FP64 oracle.

* cells of 0 to 8 and of 9 to 40 atoms: the series of a few atoms and of many;
  8, 16 and 32 lanes per near-field chunk;
* atoms outside the box beyond the series' range (the cell's circumscribed
  sphere and 2 %) and slightly outside it (within the range);
* cells of 128 and 129 atoms (a whole atom tile, and one atom of the next);
* tolerances from 1e-2 to 1e-7: 4 to 42 series terms, 2 to 41 radial nodes.

Bars: forces 1e-5 of the far field's RMS (an FP32 phase carries about |k.d| x 6e-8
<= 2e-6 rad at |k.d| <= 30 rad, the atoms far outside twice that; measured 1e-7 to
4e-7) and 1e-12 of the total for the near field's FP64 sums beside it; per-atom
energies the same; the total energy 1e-6 of the sum of its terms' magnitudes.
(The near field by itself: test_gpu_clusters.py.)
"""
import numpy as np
import pytest

from oracle import oracle, planner

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda:0")


def _points(kind):
    """(positions, box edge, rcut) of a cubic system."""
    rng = np.random.default_rng(41)
    if kind.startswith("sparse"):
        n, cells = (420, 5) if kind == "sparse_8" else (1500, 4)
        return rng.uniform(0.0, 10.0 * cells, size=(n, 3)), 10.0 * cells, 10.0
    if kind == "outside":
        pts = rng.uniform(0.0, 40.0, size=(2000, 3))
        pts[:40] = rng.uniform(-8.0, -4.0, size=(40, 3))            # beyond the range of the corner cell
        pts[40:60] = 40.0 + rng.uniform(4.0, 8.0, size=(20, 3))
        pts[60:90, 0] = -0.3                                        # outside, within the range
        return pts, 40.0, 10.0
    if kind == "tile_edges":  # 128 and 129 atoms per cell, alternately
        pts = []
        for c in range(64):
            o = 10.0 * np.array([c // 16, (c // 4) % 4, c % 4])
            pts.append(o + rng.uniform(0.01, 9.99, size=(128 + c % 2, 3)))
        return np.concatenate(pts), 40.0, 10.0
    return rng.uniform(0.0, 40.0, size=(900, 3)), 40.0, 10.0


@pytest.mark.parametrize("kind,tol", [("sparse_8", 1e-4), ("sparse_40", 1e-5), ("outside", 1e-4),
                                      ("tile_edges", 1e-4), ("uniform", 1e-2), ("uniform", 1e-3),
                                      ("uniform", 1e-6), ("uniform", 1e-7)])
def test_series_forms_match_oracle(pkg, store, kind, tol):
    pts, L, rcut = _points(kind)
    rng = np.random.default_rng(43)
    pts = pts[rng.permutation(len(pts))]
    x, y, z = (np.ascontiguousarray(pts[:, i]) for i in range(3))
    q = rng.choice([-0.834, 0.417, 0.417], len(x))
    p = planner.make_plan(len(x), tol, (L, L, L), rcut, store)
    with pkg.GlstForce(len(x), tol, L, L, L, rcut=rcut) as f:
        f.calc_ener_force(_dev(x), _dev(y), _dev(z), _dev(q))
        got = f.get_ef()
        sidx, cnt, _pnt = f.assignment()
    assert p.has_far
    near = oracle.glst(x, y, z, q, p, far=False)
    ref = oracle.glst(x, y, z, q, p)
    _ac, rcnt, _rpnt, rsidx = oracle.assign(x, y, z, p)
    assert np.array_equal(cnt, rcnt) and np.array_equal(sidx, rsidx)
    if kind == "tile_edges":
        assert sorted(set(cnt)) == [128, 129]
    # the far field by itself: what the near field (FP64, to 1e-12) leaves
    far = [r - n for r, n in zip(ref, near)]
    err = [g - r for g, r in zip(got, ref)]
    scale = np.sqrt(np.mean(sum(a * a for a in far[:3])))
    rms = np.sqrt(np.mean(sum(a * a for a in err[:3])))
    total = np.sqrt(np.mean(sum(a * a for a in ref[:3])))
    assert rms <= 1e-5 * scale + 1e-12 * total, (kind, tol, rms / scale)
    e_rms, e_far, e_total = (np.sqrt(np.mean(a[3] * a[3])) for a in (err, far, ref))
    assert e_rms <= 1e-5 * e_far + 1e-12 * e_total, (kind, tol, e_rms / e_far)
    assert abs(np.sum(err[3])) <= 1e-6 * np.sum(np.abs(ref[3])), (kind, tol)
