"""The server reserves no less than a system's handle takes.

A server whose budget is one byte below the device bytes of a system's handle
must refuse the request (its reservation is an upper bound of the handle's
size); otherwise it would allocate past its budget.  The shapes are those where
partial rows outnumber what the tile counts suggest: few tiles of several
groups (padded to quads), a ragged grid, an axis of 1,024 cells, a million atoms,
and a shape whose launches were tuned for more waves of gather warps.
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

T0 = math.erfc(3.1) / 10.0


def _refused(pkg, n, tol, box, rcut):
    rng = np.random.default_rng(3)
    x, y, z = (rng.uniform(0.0, b, n) for b in box)
    q = np.zeros(n)
    with pkg.GlstForce(n, tol, *box, rcut=rcut) as f:
        need = f.info().device_bytes
    with pkg.GlstServer(need - 1, nslots=1) as s:
        t = s.submit(1, x, y, z, q, tol, box, rcut)
        with pytest.raises(pkg.GlstError) as e:
            s.wait(t, timeout_ms=120000)
    return e.value.status == 6


@pytest.mark.parametrize("n,tol,box,rcut", [
    (90000, 1e-3, (96.5,) * 3, 8.0),
    (60000, T0, (96.5,) * 3, 14.0),
    (12000, 0.1 * T0, (30.0, 50.0, 80.0), 10.0),
    (200, 1e-4, (10240.0, 30.0, 30.0), 10.0),
    (1000000, 1e-2, (60.0,) * 3, 20.0),
])
def test_reservation_covers_the_handle(pkg, n, tol, box, rcut):
    assert _refused(pkg, n, tol, box, rcut)


def test_reservation_follows_the_tuned_shape(pkg):
    n, box = 30000, (66.9,) * 3
    rng = np.random.default_rng(4)
    dev = [torch.tensor(rng.uniform(0.0, 66.9, n), device="cuda:0") for _ in range(3)]
    dev.append(torch.zeros(n, dtype=torch.float64, device="cuda:0"))
    with pkg.GlstForce(n, T0, *box, rcut=10.0) as f:
        f.autotune(*dev)
    assert _refused(pkg, n, T0, box, 10.0)
