"""Performance cases of the GLST engine: what a program that uses it calls.

Every case is a solve -- the energies and forces of water boxes -- through the
package's public entry points: a handle with its inputs on the device
(``GlstForce.calc_ener_force`` and ``get_ef``), a handle called with host
arrays (``compute_host``), a batch of independent boxes (``GlstBatch``), and a
burst of requests to the server (``GlstServer``).  Boxes, cutoffs, tolerances
and size ranges are those of ``systems.py``, of the tests and of ``bench.py``.
"""
import importlib
import math

import numpy as np
import torch

glst = importlib.import_module("gauss-legendre-spherical-t_b200")

T0 = math.erfc(3.1) / 10.0  # alpha 0.31 / A at a 10 A cutoff: the default order
DENSITY = 0.0334            # molecules per cubic A


def _solve(name, n_mol, box, rcut, tol, ct="double", kind="solve"):
    bx, by, bz = box if isinstance(box, tuple) else (box, box, box)
    c = dict(kind=kind, n_mol=n_mol, bx=bx, by=by, bz=bz, rcut=rcut, tol=tol, ct=ct)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest system: near field only (its grid's outer layer is empty), a latency case
        _solve("water216", 216, 18.63, 9.0, math.erfc(0.34 * 9.0) / 9.0),
        # a small molecule box at the default order, 4^3 cells: an MD step of a small system
        _solve("water1000", 1000, 31.04, 10.0, T0),
        # a coarse tolerance and a short cutoff on a small box: the far field of a few thousand nodes
        _solve("water1000_coarse", 1000, 31.04, 8.0, 1e-4),
        # a ragged box: 5 x 6 x 4 cells, outer layers nearly empty, an odd atom count
        _solve("slab4003", 4003, (41.5, 58.3, 39.1), 10.0, T0),
        # the headline system: 30,000 atoms, 7^3 cells, default order
        _solve("water10k", 10000, 66.9, 10.0, T0),
        # the same at the next higher order, and binned in float (glst_force<float>)
        _solve("water10k_next_float", 10000, 66.9, 10.0, 0.1 * T0, ct="float"),
        # a long cutoff: 5^3 cells of about 170 atoms
        _solve("water7000_rcut14", 7000, 60.0, 14.0, 1e-5),
        # a dilute, wide box at a coarse tolerance: 26^3 cells of a few atoms
        _solve("wide33k_26cells", 33333, 260.0, 10.0, 1e-3),
        # the largest system: a million atoms on 22^3 cells, default order
        _solve("water333k", 333333, 215.3, 10.0, T0),
        # a program without device arrays: host inputs to host results
        _solve("host2000", 2000, 39.1, 10.0, 1e-5, kind="host"),
        # independent boxes of uneven size (300 to 30,000 atoms, two orders) in one call
        dict(name="batch48", kind="batch", n_sys=48, mol_min=100, mol_max=10000, rcut=10.0, tol=T0),
        # a burst of served requests, 60 % of them continuing resident systems
        dict(name="served10", kind="serve", n_req=10, mol_min=333, mol_max=33333, rcut=10.0, tol=T0),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["solve"] * 6 + ["host", "batch", "serve"])
    if kind == "batch":
        lo = log_int(100, 1000)
        return dict(kind=kind, n_sys=log_int(4, 40), mol_min=lo, mol_max=log_int(lo + 1, 10000), rcut=10.0, tol=T0)
    if kind == "serve":
        lo = log_int(333, 2000)
        return dict(kind=kind, n_req=rng.randint(3, 12), mol_min=lo, mol_max=log_int(lo + 1, 33333), rcut=10.0,
                    tol=T0)
    n_mol = log_int(100, 30000)
    rcut = rng.choice([8.0, 9.0, 10.0, 10.0, 12.0, 14.0])
    tol = rng.choice([1e-3, 1e-4, 1e-5, T0, T0, 0.1 * T0])
    edge = (n_mol / DENSITY) ** (1.0 / 3.0)
    a, b = (1.0, 1.0) if rng.random() < 0.5 else (rng.uniform(0.75, 1.35), rng.uniform(0.75, 1.35))
    box = (round(edge * a, 3), round(edge * b, 3), round(edge / (a * b), 3))
    return _solve(None, n_mol, box, rcut, tol, ct=rng.choice(["double", "double", "float"]), kind=kind)


# ------------------------------------------------------------------ inputs
def _water(n_mol, box, seed):
    """Rigid TIP3P-like waters (charges -0.834 and 0.417) on jittered lattice
    sites with random orientations; minimum coordinates at 0, as a driver
    recentres them.  (x, y, z, q), FP64."""
    rng = np.random.default_rng(seed)
    box = np.asarray(box, dtype=np.float64)
    s = (box.prod() / n_mol) ** (1.0 / 3.0)
    m = np.maximum(1, np.round(box / s).astype(int))
    while m.prod() < n_mol:
        m[np.argmax(box / m)] += 1
    sites = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    if len(sites) > n_mol:
        sites = sites[np.sort(rng.choice(len(sites), n_mol, replace=False))]
    o = (sites + 0.5) * (box / m) + rng.uniform(-0.3, 0.3, size=(n_mol, 3))
    # two O-H bonds of 0.9572 A at 104.52 degrees, in a random orthonormal frame
    u = rng.normal(size=(n_mol, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = np.cross(u, rng.normal(size=(n_mol, 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    half = 0.5 * math.radians(104.52)
    a, b = 0.9572 * math.cos(half) * u, 0.9572 * math.sin(half) * v
    pos = np.stack([o, o + a + b, o + a - b], axis=1).reshape(-1, 3)
    pos -= pos.min(axis=0)
    return tuple(np.ascontiguousarray(pos[:, i]) for i in range(3)) + (np.tile([-0.834, 0.417, 0.417], n_mol),)


def _systems(case, seed):
    """The case's systems: dicts of natom, tol, box, rcut, ct and pos (host arrays)."""
    if case["kind"] in ("solve", "host"):
        box = (case["bx"], case["by"], case["bz"])
        return [dict(pos=_water(case["n_mol"], box, seed), natom=3 * case["n_mol"], tol=case["tol"], box=box,
                     rcut=case["rcut"], ct=case["ct"])]
    n = case["n_sys"] if case["kind"] == "batch" else case["n_req"]
    # sizes log-uniform, the same for every seed (a case is one amount of work)
    sizes = np.random.default_rng(7)
    out = []
    for i in range(n):
        f = (i + sizes.uniform()) / n  # stratified over the range
        mol = int(round(case["mol_min"] * (case["mol_max"] / case["mol_min"]) ** f))
        edge = (mol / DENSITY) ** (1.0 / 3.0)
        tol = case["tol"] * (0.1 if case["kind"] == "batch" and i % 2 else 1.0)
        out.append(dict(pos=_water(mol, (edge,) * 3, seed * 1009 + i), natom=3 * mol, tol=tol, box=(edge,) * 3,
                        rcut=case["rcut"], ct="double"))
    order = sizes.permutation(n)
    return [out[i] for i in order]


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    systems = _systems(case, seed)
    if s.kind in ("solve", "host"):
        d = systems[0]
        s.force = glst.GlstForce(d["natom"], d["tol"], *d["box"], rcut=d["rcut"], ct=d["ct"])
        if s.kind == "host":
            s.args = d["pos"]
        else:
            s.args = [_device(a) for a in d["pos"]]
            s.out = [torch.empty(d["natom"], dtype=torch.float64, device="cuda") for _ in range(4)]
    elif s.kind == "batch":
        s.batch = glst.GlstBatch(systems)
        s.args = [_device(np.concatenate([d["pos"][k] for d in systems])) for k in range(4)]
        s.out = [torch.empty_like(s.args[0]) for _ in range(4)]
    else:
        s.server = glst.GlstServer(100 << 30, nslots=8)
        # four requests in ten name no resident system: theirs is set up and dropped again
        s.requests = [(0 if i % 5 in (1, 3) else i + 1, d) for i, d in enumerate(systems)]
    return s


def run(state):
    s = state
    if s.kind == "solve":
        s.force.calc_ener_force(*s.args)
        s.force.get_ef(*s.out)
        return s.out
    if s.kind == "host":
        return list(s.force.compute_host(*s.args)) + [s.force.energy()]
    if s.kind == "batch":
        s.batch.compute(*s.args, *s.out)
        return s.out + [s.batch.energies()]
    tickets = [s.server.submit(key, *d["pos"], d["tol"], d["box"], d["rcut"]) for key, d in s.requests]
    return [list(s.server.wait(t)[:5]) for t in tickets]


# ------------------------------------------------------- work and tolerance
_plans = {}


def _plan(d):
    """The cubature rule of a system (cells, groups, nodes and weights): the
    sum that every implementation of the method evaluates."""
    key = (d["natom"], d["tol"], d["box"], d["rcut"], d["ct"])
    if key not in _plans:
        _plans[key] = glst.plan(d["natom"], d["tol"], d["box"], d["rcut"], ct=d["ct"])
    return _plans[key]


def _sizes(case):
    if case["kind"] in ("solve", "host"):
        box = (case["bx"], case["by"], case["bz"])
        return [dict(natom=3 * case["n_mol"], tol=case["tol"], box=box, rcut=case["rcut"], ct=case["ct"])]
    return [{k: v for k, v in d.items() if k != "pos"} for d in _systems(case, 0)]


def work(case):
    """Four FP64 values in and four out per atom.  Near field: about 20
    operations for each pair of atoms in neighbouring cells, at the box's mean
    density.  Far field: one multiply-add per (atom, node) in each of the two
    passes over atoms, and for each (cell, node) two box filters along three
    axes of complex values."""
    nbytes = flops = 0.0
    for d in _sizes(case):
        inf, _ = _plan(d)
        n, (nx, ny, nz) = d["natom"], inf.ncell
        nbytes += 64.0 * n
        vol = d["box"][0] * d["box"][1] * d["box"][2]
        ranges = [min(3 * d["rcut"], b) for b in d["box"]]
        flops += 20.0 * n * (n / vol) * ranges[0] * ranges[1] * ranges[2]
        if inf.has_far_field:
            flops += 4.0 * n * inf.num_nodes + 24.0 * nx * ny * nz * inf.num_nodes
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """FP64 near field, FP32 phases and sums in the far field.  The per-atom
    energies are the widest: their far-field terms cancel.  Measured against
    ``exact``: 2e-7 to 9e-7 up to 120,000 atoms, 2.4e-6 at a million (forces
    1e-8 to 7e-8), and 6e-16 on grids without a far field."""
    if not any(_plan(d)[0].has_far_field for d in _sizes(case)):
        return dict(rel=1e-12)
    return dict(rel=4e-6 if max(d["natom"] for d in _sizes(case)) <= 200000 else 1e-5)


# ---------------------------------------------------------------- FP64 values
def _exact(d):
    """The cubature sum of one system in FP64 with torch: cells padded to the
    fullest one, near field over the 27 neighbour cells, far field over chunks
    of nodes (structure factors, box sums by prefix sums, gather)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    inf, (kx, ky, kz, w, group) = _plan(d)
    n, (nx, ny, nz) = d["natom"], tuple(inf.ncell)
    C = nx * ny * nz
    xyz = torch.from_numpy(np.stack(d["pos"][:3], 1))
    q = torch.from_numpy(d["pos"][3])
    if d["ct"] == "float":  # binned in float
        inv = torch.tensor(1.0, dtype=torch.float32) / torch.tensor(d["rcut"], dtype=torch.float32)
        b = (xyz.float() * inv).to(torch.int64)
        kx, ky, kz, w = (a.astype(np.float32).astype(np.float64) for a in (kx, ky, kz, w))
    else:
        b = (xyz * (1.0 / d["rcut"])).to(torch.int64)
    b = torch.minimum(b.clamp_min(0), torch.tensor([nx - 1, ny - 1, nz - 1]))
    cell = (b[:, 0] * ny + b[:, 1]) * nz + b[:, 2]
    order = torch.argsort(cell, stable=True)
    cnt = torch.bincount(cell, minlength=C)
    m = int(cnt.max())
    first = torch.cumsum(cnt, 0) - cnt
    sc = cell[order]
    slot = sc * m + torch.arange(n) - first[sc]  # place in the padded array
    P = torch.zeros(C * m, 4, dtype=torch.float64)
    P[slot] = torch.cat([xyz, q[:, None]], 1)[order]
    P = P.to(dev).view(C, m, 4)
    live = (torch.arange(m)[None, :] < cnt[:, None]).to(dev)
    F = torch.zeros(C, m, 4, dtype=torch.float64, device=dev)
    # near field
    ids = torch.arange(C, device=dev)
    ix, iy, iz = ids // (ny * nz), (ids // nz) % ny, ids % nz
    eye = torch.eye(m, dtype=torch.bool, device=dev)
    per = max(1, 30_000_000 // (m * m))
    for ox in (-1, 0, 1):
        for oy in (-1, 0, 1):
            for oz in (-1, 0, 1):
                jx, jy, jz = ix + ox, iy + oy, iz + oz
                ok = (jx >= 0) & (jx < nx) & (jy >= 0) & (jy < ny) & (jz >= 0) & (jz < nz)
                src = ids[ok]
                dst = ((jx * ny + jy) * nz + jz)[ok]
                for c0 in range(0, len(src), per):
                    s, t = src[c0:c0 + per], dst[c0:c0 + per]
                    use = live[s][:, :, None] & live[t][:, None, :]
                    if ox == oy == oz == 0:
                        use = use & ~eye
                    dx = P[s][:, :, None, :3] - P[t][:, None, :, :3]
                    r2 = torch.where(use, dx.square().sum(-1), 1.0)
                    e = torch.where(use, P[s][:, :, None, 3] * P[t][:, None, :, 3] / r2.sqrt(), 0.0)
                    F[s, :, 3] += e.sum(2)
                    F[s, :, :3] += ((e / r2)[..., None] * dx).sum(2)
    # far field
    if inf.has_far_field:
        K = inf.num_nodes
        kv = torch.from_numpy(np.stack([kx, ky, kz], 1)).to(dev)
        wv = torch.from_numpy(w).to(dev)
        gl = group.astype(np.int64)
        bounds = [0] + [int(v) + 1 for v in np.nonzero(np.diff(gl))[0]] + [K]

        def box_sum(a, r):
            for axis, size in enumerate((nx, ny, nz)):
                z = torch.zeros_like(a.narrow(axis, 0, 1))
                p = torch.cat([z, torch.cumsum(a, axis)], axis)
                i = torch.arange(size, device=dev)
                a = p.index_select(axis, (i + r).clamp_max(size - 1) + 1) - p.index_select(axis, (i - r).clamp_min(0))
            return a

        chunk = max(8, 100_000_000 // (C * m))
        for k_lo, k_hi in zip(bounds, bounds[1:]):
            g = int(gl[k_lo])
            r_in, r_out = int(inf.group_r_in[g]), int(inf.group_r_out[g])
            for k0 in range(k_lo, k_hi, chunk):
                k = kv[k0:min(k_hi, k0 + chunk)]
                th = (P[:, :, :3].reshape(-1, 3) @ k.T).view(C, m, -1)
                cs, sn = torch.cos(th), torch.sin(th)
                del th
                qq = P[:, None, :, 3]
                S = torch.complex((qq @ cs)[:, 0], -(qq @ sn)[:, 0]).view(nx, ny, nz, -1)
                R = (wv[k0:k0 + len(k)] * (box_sum(S, r_out) - box_sum(S, r_in))).view(C, -1)
                # q Re(e^{ik.r} R) and q Im(e^{ik.r} R) k
                a = torch.stack([R.imag * k[:, i] for i in range(3)] + [R.real], -1)
                bm = torch.stack([R.real * k[:, i] for i in range(3)] + [-R.imag], -1)
                F += P[:, :, 3:4] * (cs @ a + sn @ bm)
    out = torch.empty(n, 4, dtype=torch.float64)
    out[order] = F.view(C * m, 4).cpu()[slot]
    return [out[:, i].contiguous().numpy() for i in range(4)]


def exact(case, seed):
    systems = _systems(case, seed)
    each = [_exact(d) for d in systems]
    if case["kind"] == "solve":
        return each[0]
    if case["kind"] == "host":
        return each[0] + [0.5 * float(each[0][3].sum())]
    if case["kind"] == "batch":
        return [np.concatenate([e[k] for e in each]) for k in range(4)] + [
            np.array([0.5 * e[3].sum() for e in each])]
    return [e + [0.5 * float(e[3].sum())] for e in each]
