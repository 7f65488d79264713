"""Timed work of the library, as a time-dependent DFT program calls it.

Each case is one call (or one short chain of calls) of the public Python
mirror of the C ABI: H psi, a Taylor step with its observables or density, time
propagation, grouped systems, the adjoint of a propagation, the Lanczos
exponential, and the orthonormalisation of the states.  Systems are made from
a seed: soft-Coulomb wells, Kleinman-Bylander atoms of nine projectors (l = 0,
1, 2) on 2-bohr spheres, states of smoothed complex Gaussian noise.

``exact`` restates every call in 64-bit torch on dense grids (the star stencil
by shifted slices, the projectors by matrix products), without the library.
"""
import functools
import importlib
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "octopus-debian-package_b200")
if os.path.isdir(os.path.join(os.getcwd(), "octopus-debian-package_b200")):
    _PKG = os.path.join(os.getcwd(), "octopus-debian-package_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

lib = importlib.import_module("hpsi.lib")
mesh_mod = importlib.import_module("hpsi.mesh")
star_points = importlib.import_module("hpsi.stencil").star_points

DEV = "cuda"
ATOM_RADIUS = 2.0
# second derivative, eighth order: offsets 0..4
FD = (-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0)
LASER = dict(E0=0.01, omega=0.057, T=50.0, pol=(0.0, 0.0, 1.0))


# ---------------------------------------------------------------------------
# the cases


def _case(name, kind, shape, n, h, atoms, nst, ld, dtype, **more):
    """shape "sphere": n = radius in tenths of a bohr; "box" / "periodic": n = "nx,ny,nz" points."""
    c = dict(name=name, kind=kind, shape=shape, n=n, h=h, atoms=atoms, nst=nst, ld=ld, dtype=dtype)
    c.update(more)
    return c


def listed():
    return [
        # a production cluster run: 32 pseudo-atoms on 904,089 points, all 128 orbitals in one block
        _case("h_cluster_f64", "apply", "sphere", 120, 0.2, 32, 128, 128, "c128"),
        # the same with single-precision states
        _case("h_cluster_f32", "apply", "sphere", 120, 0.2, 32, 128, 128, "c64"),
        # one block of states of a plain box without projectors (jellium, model potentials)
        _case("h_box_f64", "apply", "box", "64,64,64", 0.25, 0, 32, 32, "c128"),
        # a small molecule on a coarse grid, a few orbitals: launches and host work count
        _case("h_molecule_f64", "apply", "sphere", 36, 0.3, 3, 6, 6, "c128"),
        # a crystal cell at a k point off Gamma: Bloch phases on the boundary and in the projectors, odd sides
        _case("h_crystal_f64", "apply", "periodic", "45,40,51", 0.3, 8, 20, 20, "c128"),
        # one real-time step with its energies, dipoles and norms, padded batch
        _case("taylor_box_f32", "taylor", "box", "57,61,66", 0.25, 6, 45, 48, "c64", dt=0.005),
        # one real-time step and the density the next potential is made from
        _case("density_step_f64", "density", "sphere", 80, 0.2, 16, 64, 64, "c128", dt=0.005),
        # real-time propagation in a laser field, steps replayed from a graph
        _case("td_cluster_f32", "td", "sphere", 120, 0.2, 32, 64, 64, "c64", dt=0.005, steps=6),
        # many uneven systems advanced together (conformers, snapshots)
        _case("group_f64", "group", "box", "", 0.25, 5, 24, 0, "c128", dt=0.005, steps=2, systems=16, side=44),
        # one control iteration of optimal control: forward, backward, gradients
        _case("control_f64", "adjoint", "box", "48,48,48", 0.25, 0, 16, 16, "c128", dt=0.01, steps=20),
        # a long step by Krylov spaces
        _case("lanczos_f64", "lanczos", "sphere", 80, 0.2, 16, 32, 32, "c128", dt=0.05),
        # re-orthonormalisation of the orbitals and their overlap matrix
        _case("orthonormalise_f64", "orthonormalise", "sphere", 80, 0.2, 0, 96, 96, "c128"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "taylor", "density", "td", "group", "adjoint", "lanczos",
                       "orthonormalise"])
    dtype = rng.choice(["c128", "c64"])
    if kind in ("adjoint", "lanczos"):
        dtype = "c128"
    if kind == "group":
        return dict(kind=kind, shape="box", n="", h=0.25, atoms=rng.randint(2, 6), nst=int(_log(rng, 4, 40)), ld=0,
                    dtype=dtype, dt=0.005, steps=2, systems=rng.randint(3, 16), side=rng.randint(32, 48))
    most = {"apply": 904000, "taylor": 300000, "density": 300000, "td": 300000, "adjoint": 90000, "lanczos": 200000,
            "orthonormalise": 300000}[kind]
    points = _log(rng, 6000, most)
    if kind == "adjoint":
        nst = int(_log(rng, 2, 20))
    else:
        nst = int(min(128, _log(rng, 3, 129), max(3, 6e7 / points)))
    pad = rng.choice([2, 4, 8]) if dtype == "c128" else rng.choice([4, 8, 16])
    ld = -(-nst // pad) * pad
    shape = rng.choice(["sphere", "box"] + (["periodic"] if kind in ("apply", "taylor") else []))
    h = rng.choice([0.2, 0.25, 0.3])
    atoms = rng.choice([0, 1]) * max(1, min(32, int(points * h ** 3 / 150.0)))
    if shape == "sphere":
        n = max(30, int(10 * h * (points * 3 / (4 * math.pi)) ** (1 / 3)))
    else:
        s = points ** (1 / 3)
        a, b = rng.uniform(0.8, 1.25), rng.uniform(0.8, 1.25)
        n = ",".join(str(max(14, int(v))) for v in (s * a, s * b, s / (a * b)))
    c = dict(kind=kind, shape=shape, n=n, h=h, atoms=atoms, nst=nst, ld=ld, dtype=dtype)
    if kind in ("adjoint",):
        c.update(dt=0.005, steps=rng.randint(6, 20))
        c["atoms"] = 0
    elif kind == "td":
        c.update(dt=0.005, steps=rng.randint(2, 6))
    elif kind == "lanczos":
        c.update(dt=0.02)
    elif kind == "orthonormalise":
        c["atoms"] = 0
    elif kind in ("taylor", "density"):
        c.update(dt=0.005)
    return c


# ---------------------------------------------------------------------------
# systems


@functools.lru_cache(maxsize=40)
def _mesh(shape, n, h):
    if shape == "sphere":
        return mesh_mod.sphere_mesh(n / 10.0, h)
    sides = tuple(int(s) for s in n.split(","))
    return mesh_mod.index_box_mesh(sides, h, periodic=shape == "periodic")


def _weights(h):
    """The star's 25 weights in the order of star_points: x with the centre, then y and z."""
    w = []
    for axis in range(3):
        for d in range(-4, 5):
            if d or axis == 0:
                w.append((FD[abs(d)] if d else 3 * FD[0]) / h ** 2)
    return np.asarray(w)


class _Projectors:
    def __init__(self, maps, mats, scals):
        self.maps, self.mats, self.scals = maps, mats, scals


def _harmonics(x, y, z, r2):
    r = np.sqrt(np.where(r2 < 1e-30, 1.0, r2))
    x, y, z = x / r, y / r, z / r
    c0, c1, c2 = 0.5 / math.sqrt(math.pi), math.sqrt(3 / (4 * math.pi)), math.sqrt(15 / (4 * math.pi))
    out = np.stack([np.full_like(x, c0), c1 * x, c1 * y, c1 * z, c2 * x * y, c2 * y * z, c2 * x * z,
                    0.5 * c2 * (x * x - y * y), 0.5 * c2 / math.sqrt(3.0) * (3 * z * z - 1)], axis=1)
    out[r2 < 1e-30, 1:] = 0.0
    return out


class _System:
    """Mesh, potential and projectors of one seed (host arrays)."""

    def __init__(self, shape, n, h, atoms, seed):
        rng = np.random.default_rng(seed)
        m = self.mesh = _mesh(shape, n, h)
        self.h, self.periodic = h, shape == "periodic"
        inner = m.lxyz[: m.np]
        lo, hi = inner.min(axis=0) * h, inner.max(axis=0) * h
        c, half = (lo + hi) / 2, (hi - lo) / 2
        x = torch.from_numpy(inner).to(DEV).double() * h
        v = torch.zeros(m.np, dtype=torch.float64, device=DEV)
        for _ in range(8):
            z = rng.uniform(1.0, 4.0)
            p = torch.as_tensor(c + rng.uniform(-0.6, 0.6, 3) * half, device=DEV)
            v -= z / torch.sqrt(((x - p) ** 2).sum(dim=1) + 1.0)
        self.v = v.cpu().numpy()
        self.proj = None
        self.k = np.array([0.21, -0.13, 0.34]) / h * 0.25 if self.periodic else None
        if atoms:
            self.proj = self._atoms(rng, atoms, c, half, shape == "sphere")
        self.phase_corr = self.kb_phases = None
        if self.periodic:
            d = (m.lxyz[m.np:] - m.lxyz[m.per_inner]) * h
            self.phase_corr = np.exp(1j * (d @ self.k))
            if self.proj is not None:
                self.kb_phases = [np.exp(-1j * ((inner[mp] * h) @ self.k)) for mp in self.proj.maps]

    def _atoms(self, rng, atoms, c, half, round_):
        m, h = self.mesh, self.h
        inner = m.lxyz[: m.np]
        l0 = inner.min(axis=0)
        ext = inner.max(axis=0) - l0 + 1
        lut = -np.ones(ext, dtype=np.int32)
        lut[tuple((inner - l0).T)] = np.arange(m.np, dtype=np.int32)
        room = np.maximum(half - ATOM_RADIUS, 0.3 * half)
        pos, tries, dist = [], 0, 2.5
        while len(pos) < atoms:
            tries += 1
            if tries % 2000 == 0:
                dist *= 0.9
            u = rng.uniform(-1.0, 1.0, 3)
            if round_ and u @ u > 1.0:
                continue
            p = c + u * room
            if all(np.linalg.norm(p - q) >= dist for q in pos):
                pos.append(p)
        maps, mats, scals = [], [], []
        for p in pos:
            a = np.maximum(np.ceil((p - ATOM_RADIUS) / h).astype(int), l0)
            b = np.minimum(np.floor((p + ATOM_RADIUS) / h).astype(int), l0 + ext - 1)
            g = np.stack(np.meshgrid(*[np.arange(a[d], b[d] + 1) for d in range(3)], indexing="ij"), -1).reshape(-1, 3)
            row = lut[tuple((g - l0).T)]
            d = g * h - p
            r2 = (d * d).sum(axis=1)
            keep = (row >= 0) & (r2 <= ATOM_RADIUS ** 2)
            order = np.argsort(row[keep])
            d, r2, row = d[keep][order], r2[keep][order], row[keep][order]
            mat = np.exp(-r2 / 0.8)[:, None] * _harmonics(d[:, 0], d[:, 1], d[:, 2], r2)
            maps.append(row.astype(np.int32))
            mats.append(np.ascontiguousarray(mat))
            scals.append(rng.uniform(-2.0, 2.0, mat.shape[1]) * h ** 3)
        return _Projectors(maps, mats, scals)

    def states(self, nst, ld, rows, seed, dtype):
        """(rows, ld) states: complex Gaussian noise, a 3-point filter along each axis, unit norm."""
        m = self.mesh
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) * 7919 + 17)
        inner = torch.from_numpy(m.lxyz[: m.np]).to(DEV).long()
        l0, l1 = inner.min(dim=0).values, inner.max(dim=0).values
        ext = [int(e) + 3 for e in (l1 - l0)]
        at = inner - l0 + 1
        out = torch.zeros((rows, ld), dtype=dtype, device=DEV)
        step = max(1, min(nst, int(2e9 // (16 * ext[0] * ext[1] * ext[2]))))
        for s in range(0, nst, step):
            e = min(nst, s + step)
            f = torch.randn((m.np, e - s, 2), generator=g, dtype=torch.float64, device=DEV)
            grid = torch.zeros(ext + [e - s], dtype=torch.complex128, device=DEV)
            grid[at[:, 0], at[:, 1], at[:, 2]] = torch.view_as_complex(f)
            for ax in range(3):
                t = grid.clone()
                n = ext[ax]
                t.narrow(ax, 1, n - 1).add_(grid.narrow(ax, 0, n - 1))
                t.narrow(ax, 0, n - 1).add_(grid.narrow(ax, 1, n - 1))
                grid = t
            y = grid[at[:, 0], at[:, 1], at[:, 2]]
            y /= (y.abs().square().sum(dim=0) * self.h ** 3).sqrt()
            out[: m.np, s:e] = y.to(dtype)
        return out


def _dtype(case):
    return torch.complex128 if case["dtype"] == "c128" else torch.complex64


def _group_sizes(case):
    """Sides and state counts of the grouped systems: around the case's own, uneven."""
    r = np.random.default_rng(case["systems"] * 1000 + case["side"])
    sides = np.clip((case["side"] * np.exp(r.uniform(-0.35, 0.35, case["systems"]))).astype(int), 24, 72)
    nsts = np.clip((case["nst"] * np.exp(r.uniform(-1.0, 0.6, case["systems"]))).astype(int), 3, 64)
    return [(int(s), int(n)) for s, n in zip(sides, nsts)]


def _systems(case, seed):
    """[(system, nst, ld)] of a case."""
    if case["kind"] == "group":
        return [(_System("box", f"{s},{s},{s}", case["h"], case["atoms"], seed * 100 + i), n, 8 * -(-n // 8))
                for i, (s, n) in enumerate(_group_sizes(case))]
    return [(_System(case["shape"], case["n"], case["h"], case["atoms"], seed), case["nst"], case["ld"])]


def _amplitudes(case, seed):
    return np.random.default_rng(seed + 5).normal(0.0, 0.005, case["steps"])


def _occupations(case, seed):
    return np.random.default_rng(seed + 6).uniform(0.0, 2.0, case["nst"])


# ---------------------------------------------------------------------------
# the library's side


def prepare(case, seed):
    st = {"case": case, "hams": [], "psi": []}
    dt = _dtype(case)
    systems = _systems(case, seed)
    for i, (s, nst, ld) in enumerate(systems):
        dm = lib.DeviceMesh(s.mesh)
        ham = lib.Hamiltonian(dm, _weights(s.h), star_points(), v=s.v, projectors=s.proj)
        if s.phase_corr is not None:
            ham.set_phase_corr(s.phase_corr)
        if s.kb_phases is not None:
            ham.set_projector_phases(s.kb_phases)
        st["hams"].append(ham)
        st["psi"].append(s.states(nst, ld, s.mesh.np_part, seed * 31 + i, dt))
    s = st["hams"][0].dmesh
    kind = case["kind"]
    st["mesh"] = s
    if kind == "apply":
        st["out"] = torch.zeros((s.mesh.np, case["ld"]), dtype=dt, device=DEV)
    elif kind == "density":
        st["occ"] = _occupations(case, seed)
        st["rho"] = torch.zeros(s.mesh.np, dtype=torch.float64, device=DEV)
    elif kind == "group":
        st["group"] = lib.Group(st["hams"])
    elif kind == "adjoint":
        st["eps"] = _amplitudes(case, seed)
        st["target"] = systems[0][0].states(case["nst"], case["ld"], s.mesh.np_part, seed * 31 + 13, dt)
    return st


def run(st):
    case, ham, psi = st["case"], st["hams"][0], st["psi"][0]
    kind, nst = case["kind"], case["nst"]
    if kind == "apply":
        ham.apply(psi, st["out"], nst=nst)
        return st["out"]
    if kind == "taylor":
        e, d, n = ham.taylor_step(psi, case["dt"], nst=nst, observables=True)
        return {"psi": psi, "energy": e, "dipole": d, "norm": n}
    if kind == "density":
        ham.taylor_step_density(psi, case["dt"], st["occ"], rho=st["rho"], nst=nst)
        return {"psi": psi, "rho": st["rho"]}
    if kind == "td":
        e, d, n = ham.td_propagate(psi, case["steps"], case["dt"], nst=nst, graph=True, **LASER)
        return {"psi": psi, "energy": e, "dipole": d, "norm": n}
    if kind == "group":
        st["group"].taylor_steps(st["psi"], case["steps"], case["dt"], graph=True)
        return st["psi"]
    if kind == "adjoint":
        J, ge, gv, gc = ham.adjoint_gradient(psi, st["target"], st["eps"], case["dt"], ckpt=5)
        return {"J": J, "eps": ge, "v": gv, "continuous": gc}
    if kind == "lanczos":
        m, _ = ham.lanczos_step(psi, case["dt"], max_order=40, tol=1e-8, nst=nst)
        return {"psi": psi, "dimension": m}
    ham.dmesh.orthonormalize_cholesky(psi, nst=nst)
    return {"psi": psi, "overlap": ham.dmesh.dotp_matrix(psi, psi, nst=nst)}


# ---------------------------------------------------------------------------
# the least work


def work(case):
    size = 16 if case["dtype"] == "c128" else 8
    total = {"bytes": 0.0, "flops": 0.0}
    if case["kind"] == "group":
        parts = [(s ** 3, n, case["atoms"]) for s, n in _group_sizes(case)]
    else:
        if case["shape"] == "sphere":
            p = 4 / 3 * math.pi * (case["n"] / 10 / case["h"]) ** 3
        else:
            p = float(np.prod([int(s) for s in case["n"].split(",")]))
        parts = [(p, case["nst"], case["atoms"])]
    for p, nst, atoms in parts:
        sphere = 4 / 3 * math.pi * (ATOM_RADIUS / case["h"]) ** 3
        # 25 real weights times a complex number, nine projectors there and back
        h_flops = p * nst * 25 * 4 + 2 * atoms * sphere * 9 * nst * 4
        batch, kind = p * nst * size, case["kind"]
        if kind == "apply":
            b, f = 2 * batch + 8 * p, h_flops
        elif kind in ("taylor", "density"):
            b, f = 2 * batch + 8 * p, 4 * h_flops
        elif kind in ("td", "group"):
            b, f = 2 * batch + 8 * p, 4 * h_flops * case["steps"]
        elif kind == "adjoint":
            # forward and backward Taylor steps, and H^m psi of each step again for its products
            b, f = 2 * batch + 16 * p, 11 * h_flops * case["steps"]
        elif kind == "lanczos":
            b, f = 2 * batch + 8 * p, 10 * h_flops
        else:
            # overlap matrix twice (one triangle each), triangular update
            b, f = 2 * batch, 3 * p * nst * nst * 4
        total["bytes"] += b
        total["flops"] += f
    return total


def tolerance(case):
    """About four times what two orders of summation and the 64-bit restatement differ by."""
    if case["dtype"] == "c64":
        return {"rel": 8e-7, "max": 8e-6}
    if case["kind"] in ("adjoint", "lanczos"):
        return {"rel": 5e-14, "max": 5e-13}
    return {"rel": 4e-15, "max": 4e-14}


# ---------------------------------------------------------------------------
# 64-bit restatement


class _Dense:
    """H of one system on dense grids, states last."""

    def __init__(self, s):
        self.s = s
        m = s.mesh
        inner = torch.from_numpy(m.lxyz[: m.np]).to(DEV).long()
        self.l0 = inner.min(dim=0).values
        self.ext = [int(e) + 1 for e in (inner.max(dim=0).values - self.l0)]
        self.at = tuple((inner - self.l0).T)
        self.v = torch.from_numpy(s.v).to(DEV)
        self.r = [inner[:, d].double() * s.h for d in range(3)]
        w = [f / s.h ** 2 for f in FD]
        self.w = w
        self.kb = []
        if s.proj is not None:
            for i, (mp, mat, sc) in enumerate(zip(s.proj.maps, s.proj.mats, s.proj.scals)):
                ph = torch.ones(len(mp), dtype=torch.complex128, device=DEV)
                if s.kb_phases is not None:
                    ph = torch.from_numpy(s.kb_phases[i]).to(DEV)
                self.kb.append((torch.from_numpy(mp).to(DEV).long(), torch.from_numpy(mat).to(DEV).to(torch.complex128),
                                torch.from_numpy(sc).to(DEV), ph))

    def apply(self, x, field=None):
        """H x of (np, n) complex128, with v + field . r."""
        out = torch.empty_like(x)
        cells = np.prod([e + 8 for e in self.ext])
        step = max(1, int(4e9 // (16 * cells)))
        for a in range(0, x.shape[1], step):
            out[:, a:a + step] = self._star(x[:, a:a + step])
        v = self.v if field is None else self.v + sum(f * r for f, r in zip(field, self.r))
        out += v[:, None] * x
        for mp, mat, sc, ph in self.kb:
            t = sc[:, None] * (mat.T @ (x[mp] * ph[:, None]))
            out[mp] += (mat @ t) * ph.conj()[:, None]
        return out

    def _star(self, x):
        e = self.ext
        g = torch.zeros([n + 8 for n in e] + [x.shape[1]], dtype=torch.complex128, device=DEV)
        c = g[4:-4, 4:-4, 4:-4]
        c[self.at] = x
        if self.s.periodic:
            for ax in range(3):
                n = e[ax]
                ph = complex(np.exp(1j * self.s.k[ax] * n * self.s.h))
                core = [slice(4, -4)] * 3
                for side, src, f in ((slice(0, 4), slice(n, n + 4), ph.conjugate()),
                                     (slice(n + 4, n + 8), slice(4, 8), ph)):
                    to, frm = list(core), list(core)
                    to[ax], frm[ax] = side, src
                    g[tuple(to)] = g[tuple(frm)] * f
        y = c * (3 * self.w[0])
        for ax in range(3):
            n = e[ax]
            core = [slice(4, -4)] * 3
            for d in range(1, 5):
                lo, hi = list(core), list(core)
                lo[ax], hi[ax] = slice(4 - d, 4 - d + n), slice(4 + d, 4 + d + n)
                y += self.w[d] * (g[tuple(lo)] + g[tuple(hi)])
        return -0.5 * y[self.at]

    def taylor(self, x, dt, field=None, order=4):
        y, t = x.clone(), x
        for k in range(1, order + 1):
            t = self.apply(t, field) * (-1j * dt / k)
            y += t
        return y

    def observables(self, x, field=None, hx=None):
        hx = self.apply(x, field) if hx is None else hx
        dv = self.s.h ** 3
        n = x.abs().square()
        return dv * (x.conj() * hx).real.sum(dim=0), dv * (n * self.r[2][:, None]).sum(dim=0), dv * n.sum(dim=0)


def _padded(y, like_rows, ld, dtype=torch.complex128):
    out = torch.zeros((like_rows, ld), dtype=dtype, device=DEV)
    out[: y.shape[0], : y.shape[1]] = y
    return out


def _laser(t):
    if t < 0 or t > LASER["T"]:
        return 0.0
    return LASER["E0"] * math.sin(math.pi * t / LASER["T"]) ** 2 * math.cos(LASER["omega"] * t)


def exact(case, seed):
    parts = _systems(case, seed)
    dt = _dtype(case)
    if case["kind"] == "group":
        out = []
        for i, (s, nst, ld) in enumerate(parts):
            d = _Dense(s)
            x = s.states(nst, ld, s.mesh.np, seed * 31 + i, dt)[:, :nst].to(torch.complex128)
            for _ in range(case["steps"]):
                x = d.taylor(x, case["dt"])
            out.append(_padded(x, s.mesh.np_part, ld))
        return out
    s, nst, ld = parts[0]
    d, m, kind = _Dense(s), s.mesh, case["kind"]
    x = s.states(nst, ld, m.np, seed * 31, dt)[:, :nst].to(torch.complex128)
    if kind == "apply":
        return _padded(d.apply(x), m.np, ld)
    if kind == "taylor":
        e, q, n = d.observables(x)
        return {"psi": _padded(d.taylor(x, case["dt"]), m.np_part, ld), "energy": e, "dipole": q, "norm": n}
    if kind == "density":
        y = d.taylor(x, case["dt"])
        rho = (y.abs().square() * torch.from_numpy(_occupations(case, seed)).to(DEV)).sum(dim=1)
        return {"psi": _padded(y, m.np_part, ld), "rho": rho}
    if kind == "td":
        obs, step = [], case["dt"]
        for i in range(case["steps"]):
            obs.append([float(o.sum()) for o in d.observables(x, (0.0, 0.0, _laser(i * step)))])
            x = d.taylor(x, step, (0.0, 0.0, _laser((i + 0.5) * step)))
        e, q, n = np.asarray(obs).T
        return {"psi": _padded(x, m.np_part, ld), "energy": e, "dipole": q, "norm": n}
    if kind == "lanczos":
        return {"psi": _padded(d.taylor(x, case["dt"], order=64), m.np_part, ld), "dimension": None}
    if kind == "adjoint":
        return _exact_adjoint(case, seed, s, d, x)
    dv = s.h ** 3
    u = torch.linalg.cholesky(dv * (x.conj().T @ x), upper=True)
    y = torch.linalg.solve_triangular(u, x, upper=True, left=False)
    return {"psi": _padded(y, m.np_part, ld), "overlap": dv * (y.conj().T @ y)}


def _exact_adjoint(case, seed, s, d, x):
    dv, dt, eps = s.h ** 3, case["dt"], _amplitudes(case, seed)
    phi = s.states(case["nst"], case["ld"], s.mesh.np, seed * 31 + 13, _dtype(case))[:, : case["nst"]]
    phi = phi.to(torch.complex128)
    path = [x]
    for f in eps:
        path.append(d.taylor(path[-1], dt, (0.0, 0.0, float(f))))
    ov = dv * (phi.conj() * path[-1]).sum(dim=0)
    lam = phi * ov
    c = [(-1j * dt) ** k / math.factorial(k) for k in range(5)]
    z = d.r[2][:, None]
    ge, gc, gv = np.zeros(len(eps)), np.zeros(len(eps)), torch.zeros(s.mesh.np, dtype=torch.float64, device=DEV)
    for n in range(len(eps) - 1, -1, -1):
        field = (0.0, 0.0, float(eps[n]))
        hp, hl = [path[n]], [lam]
        for _ in range(3):
            hp.append(d.apply(hp[-1], field))
            hl.append(d.apply(hl[-1], field))
        t = torch.zeros_like(gv)
        for j in range(4):
            for k in range(4 - j):
                t += 2 * dv * (c[j + k + 1] * hl[j].conj() * hp[k]).real.sum(dim=1)
        gv += t
        ge[n] = float((t * z[:, 0]).sum())
        gc[n] = float((2 * dv * c[1] * (lam.conj() * z * path[n]).sum()).real)
        lam = d.taylor(lam, -dt, field)
    return {"J": float(ov.abs().square().sum()), "eps": ge, "v": gv.cpu().numpy(), "continuous": gc}
