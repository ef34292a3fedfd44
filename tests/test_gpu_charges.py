"""GPU parity where the charges are ordered: their far-field terms cancel (rock
salt), add up plane by plane (layers), or all add up (one sign).

Bars, against the FP64 oracle: forces and per-atom energies 2e-6 of the larger of
the system's own far field and that of random signs on the same sites (an FP32
phase of up to 30 rad carries 30 x 2^-24 = 2e-6 rad of every term; where terms
cancel the error does not); total energy 2^-24 of the sum of the energies'
magnitudes (one FP32 rounding of every term, all the same way).
"""
import numpy as np
import pytest

from oracle import oracle, planner

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _signs(kind, lat, rng):
    if kind == "rock_salt":
        return np.where(lat.sum(1) % 2 == 0, 1.0, -1.0)
    if kind == "layers":
        return np.where(lat[:, 0] % 2 == 0, 1.0, -1.0)
    if kind == "one_sign":
        return np.ones(len(lat))
    return rng.choice([-1.0, 1.0], len(lat))


def _rms(a):
    return np.sqrt(np.mean(sum(v * v for v in a)))


@pytest.mark.parametrize("n_axis,tol", [(16, 1e-5), (16, 1e-3), (20, 1e-4)])
def test_ordered_charges_match_the_oracle(pkg, store, n_axis, tol):
    rng = np.random.default_rng(17)
    lat = np.stack(np.meshgrid(*[np.arange(n_axis)] * 3, indexing="ij"), -1).reshape(-1, 3)
    L, rcut = 2.5 * n_axis, 10.0
    p = (lat + 0.5) * 2.5 + rng.uniform(-0.1, 0.1, lat.shape)
    x, y, z = (np.ascontiguousarray(p[:, i]) for i in range(3))
    plan = planner.make_plan(len(x), tol, (L, L, L), rcut, store)
    scale = None
    with pkg.GlstForce(len(x), tol, L, L, L, rcut=rcut) as f:
        for kind in ("random", "rock_salt", "layers", "one_sign"):
            q = _signs(kind, lat, rng)
            f.calc_ener_force(*[torch.tensor(v, device="cuda:0") for v in (x, y, z, q)])
            got = f.get_ef()
            ref = oracle.glst(x, y, z, q, plan)
            far = [r - n for r, n in zip(ref, oracle.glst(x, y, z, q, plan, far=False))]
            if scale is None:
                scale = _rms(far[:3]), _rms(far[3:])
            err = [g - r for g, r in zip(got, ref)]
            rep = (kind, _rms(err[:3]) / _rms(far[:3]), _rms(err[3:]) / _rms(far[3:]),
                   np.sum(err[3]) / np.sum(np.abs(ref[3])))
            assert _rms(err[:3]) <= 2e-6 * max(scale[0], _rms(far[:3])), rep
            assert _rms(err[3:]) <= 2e-6 * max(scale[1], _rms(far[3:])), rep
            assert abs(np.sum(err[3])) <= 2.0**-24 * np.sum(np.abs(ref[3])), rep
