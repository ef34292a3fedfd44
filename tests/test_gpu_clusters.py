"""GPU parity and speed of unevenly filled grids: atoms of a dense cell beyond
the cell's own warps' share (2.5 times the mean, in whole 32s) are listed as
pieces of 32 and taken by further warps.

* counts at the edges of the share and of the pieces (32 and 33, 64 and 65, a
  whole 128-atom tile and one more), the rest of the grid nearly empty, alone and
  in a work-list batch (bitwise the same), against the FP64 oracle: the far
  field's forces to 1e-5 of the far field (an FP32 phase of up to 30 rad carries
  2e-6 rad), per-atom energies to 1e-5 of theirs, the near field in FP64;
* near-field grids (two cells per axis), FP64 throughout: 1e-13 of the RMS force
  and energy (a sum of some hundred terms of 1e-16, the largest a few times the RMS);
* the same dense cell in a small and in a large empty box: its near field takes
  the same work, and no more than 2.5 times as long.
"""
import numpy as np
import pytest

from oracle import oracle, planner

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

COUNTS = [1, 2, 31, 32, 33, 34, 63, 64, 65, 96, 97, 128, 129, 160, 161, 300]


def _dev(a):
    return [torch.tensor(np.asarray(v), dtype=torch.float64, device="cuda:0") for v in a]


def _cluster(n_axis, seed):
    """Cells of COUNTS atoms at random places of an n_axis^3 grid of 10 A cells."""
    rng = np.random.default_rng(seed)
    cells = rng.choice(n_axis ** 3, len(COUNTS), replace=False)
    pts = []
    for c, n in zip(cells, COUNTS):
        m = int(np.ceil(n ** (1 / 3)))
        lat = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        o = 10.0 * np.array([c // n_axis ** 2, c // n_axis % n_axis, c % n_axis])
        pts.append(o + (lat + 0.5 + rng.uniform(-0.3, 0.3, lat.shape)) * 9.9 / m)
    p = np.concatenate(pts)[rng.permutation(sum(COUNTS))]
    return tuple(np.ascontiguousarray(p[:, i]) for i in range(3)) + (rng.choice([-0.834, 0.417, 0.417], len(p)),)


@pytest.mark.parametrize("n_axis,tol", [(4, 1e-4), (6, 1e-5)])
def test_dense_cells_match_the_oracle(pkg, store, n_axis, tol):
    L, rcut = 10.0 * n_axis, 10.0
    x, y, z, q = _cluster(n_axis, 5 + n_axis)
    p = planner.make_plan(len(x), tol, (L, L, L), rcut, store)
    with pkg.GlstForce(len(x), tol, L, L, L, rcut=rcut) as f:
        f.calc_ener_force(*_dev((x, y, z, q)))
        got = f.get_ef()
        energy = f.energy()
        _s, cnt, _p = f.assignment()
    assert sorted(c for c in cnt if c) == COUNTS
    near = oracle.glst(x, y, z, q, p, far=False)
    ref = oracle.glst(x, y, z, q, p)

    def rms(a):
        return np.sqrt(np.mean(sum(v * v for v in a)))
    far = [r - n for r, n in zip(ref, near)]
    err = [g - r for g, r in zip(got, ref)]
    assert rms(err[:3]) <= 1e-5 * rms(far[:3]) + 1e-12 * rms(ref[:3])
    assert rms(err[3:]) <= 1e-5 * rms(far[3:]) + 1e-12 * rms(ref[3:])
    # alone and in a batch, one launch per phase
    systems = [dict(natom=len(x), tol=tol, box=(L, L, L), rcut=rcut)] * 2
    out = [torch.empty(2 * len(x), dtype=torch.float64, device="cuda:0") for _ in range(4)]
    with pkg.GlstBatch(systems) as b:
        b.compute(*_dev(np.concatenate([v, v]) for v in (x, y, z, q)), *out, mode="worklist")
        assert np.all(np.asarray(b.energies()) == energy)
    for o, g in zip(out, got):
        assert np.array_equal(o.cpu().numpy(), np.concatenate([g, g]))


@pytest.mark.parametrize("counts", [[300, 1, 0, 2, 0, 0, 33, 0], [97, 97, 0, 0, 0, 0, 0, 1], [0, 0, 0, 0, 0, 0, 0, 129],
                                    [40, 30, 20, 10, 9, 8, 17, 16]])
def test_near_field_of_uneven_cells(pkg, store, counts):
    rng = np.random.default_rng(sum(counts))
    pts = []
    for c, n in enumerate(counts):
        m = max(1, int(np.ceil(n ** (1 / 3))))
        lat = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        pts.append(10.0 * np.array([c // 4, c // 2 % 2, c % 2]) + (lat + 0.5 + rng.uniform(-0.3, 0.3, lat.shape)) * 9.9 / m)
    p = np.concatenate(pts)[rng.permutation(sum(counts))]
    x, y, z = (np.ascontiguousarray(p[:, i]) for i in range(3))
    q = rng.choice([-0.834, 0.417, 0.417], len(p))
    plan = planner.make_plan(len(p), 1e-4, (20.0,) * 3, 10.0, store)
    assert not plan.has_far
    ref = oracle.glst(x, y, z, q, plan)
    with pkg.GlstForce(len(p), 1e-4, 20.0, 20.0, 20.0, rcut=10.0) as f:
        f.calc_ener_force(*_dev((x, y, z, q)))
        got = f.get_ef()
    for part in (slice(0, 3), slice(3, 4)):
        err = np.sqrt(np.mean(sum((g - r) ** 2 for g, r in zip(got[part], ref[part]))))
        assert err <= 1e-13 * np.sqrt(np.mean(sum(r * r for r in ref[part]))), err


def test_a_dense_cell_costs_the_same_in_a_wide_box(pkg):
    rng = np.random.default_rng(9)
    m = 20
    lat = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = 30.0 + (lat + 0.5 + rng.uniform(-0.2, 0.2, lat.shape)) * 10.0 / m
    atoms = _dev(tuple(p.T) + (rng.choice([-0.5, 0.5], len(p)),))
    ms = []
    for L in (70.0, 260.0):
        with pkg.GlstForce(len(p), 1e-3, L, L, L, rcut=10.0) as f:
            f.assign_atoms(*atoms)
            t = []
            for _ in range(4):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                f.calc_sr_ef()
                e1.record()
                torch.cuda.synchronize()
                t.append(e0.elapsed_time(e1))
            ms.append(min(t))
    assert ms[1] <= 2.5 * ms[0], ms
