"""The tensor-memory pass at the edges of its tiles, chunks and z blocks.

Sides of 16, 17 and 33 cells (whole, one-cell and two tiles), widths around the
chunk of 8 (FP64) or 16 (FP32) states (the last chunk is partial), z blocks of
a few planes, the three load maps, a laser field and complex time steps,
against the CPU oracle; grouped systems of unequal spacings and with Bloch
phases against single ones; the KB ket at every width of its blocks against a
numpy restatement.  FP64 to 1e-12 relative max-norm per state, FP32 to 2e-5 (the
parity bounds of the other passes)."""
import numpy as np
import pytest

from helpers import rel_maxnorm_per_state

pytestmark = pytest.mark.gpu

TMEM = {"c128": ("HPSI_PASS_SHAPE64", "8,2,{zb},9,1,2,0,8,0,0,0,1"),
        "c64": ("HPSI_PASS_SHAPE32", "16,2,{zb},9,1,2,1,8,0,0,0,1")}
TOL = {"c128": 1e-12, "c64": 2e-5}


def _states(m, nst, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros((m.np_part, nst), dtype=np.complex128)
    x[: m.np] = rng.standard_normal((m.np, nst)) + 1j * rng.standard_normal((m.np, nst))
    return x


def _ham(m, v=None, proj=None):
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    return lib.Hamiltonian(lib.DeviceMesh(m), laplacian_weights(m.spacing), star_points(), v=v, projectors=proj)


def _oracle(m, v=None, **more):
    from hpsi.stencil import laplacian_weights, star_points
    from oracle import oracle as O
    return O.Hamiltonian(m, laplacian_weights(m.spacing), star_points(), v=v, **more)


@pytest.mark.parametrize("zb", [0, 1, 2, 3, 4, 5, 100])
@pytest.mark.parametrize("shape", [(16, 17, 9), (33, 15, 6), (5, 4, 12)])
@pytest.mark.parametrize("dtype,nst", [("c128", 1), ("c128", 8), ("c128", 13), ("c64", 2), ("c64", 16), ("c64", 22)])
def test_tile_and_chunk_edges(cuda, dtype, nst, shape, zb, monkeypatch):
    import torch
    from hpsi import fixtures
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh(shape, 0.3)
    v = fixtures.soft_coulomb(m, np.random.default_rng(5))
    psi = _states(m, nst, 7)
    var, s = TMEM[dtype]
    monkeypatch.setenv(var, s.format(zb=zb))
    H, ref = _ham(m, v), _oracle(m, v, bc="zero")
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    x = torch.from_numpy(psi).to(cuda).to(tdt)
    y = torch.full((m.np, nst), float("nan"), dtype=tdt, device=cuda)
    H.apply(x, y)
    hx = ref.apply(psi)
    assert rel_maxnorm_per_state(y.cpu().numpy(), hx) <= TOL[dtype]
    H.apply(x, y, set_bc=False)  # stored boundary rows (zero here)
    assert rel_maxnorm_per_state(y.cpu().numpy(), hx) <= TOL[dtype]
    # Horner pass, imaginary and complex factors
    for a in (-0.01j, 0.004 - 0.01j):
        out = torch.full_like(y, float("nan"))
        H.apply_horner(x, x[: m.np].clone(), out, a)
        assert rel_maxnorm_per_state(out.cpu().numpy(), psi[: m.np] + a * hx) <= TOL[dtype]
    assert H.status() == 0


@pytest.mark.parametrize("dtype,nst", [("c128", 3), ("c128", 10), ("c64", 6), ("c64", 20)])
def test_observables_and_field(cuda, dtype, nst):
    """Energies, dipoles and norms of a first pass with a field, partial chunk."""
    import torch
    from hpsi import fixtures
    from hpsi.mesh import sphere_mesh
    m = sphere_mesh(3.2, 0.3)
    v = fixtures.soft_coulomb(m, np.random.default_rng(6))
    psi = _states(m, nst, 8)
    pol, amp = np.array([0.3, -0.5, 0.8]), 0.07
    H = _ham(m, v)
    H.set_field(pol, amp)
    r = m.x[: m.np] @ pol
    hx = _oracle(m, v + amp * r, bc="zero").apply(psi)
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    x = torch.from_numpy(psi).to(cuda).to(tdt)
    e, d, n = H.taylor_step(x.clone(), 0.002, observables=True)
    p = psi[: m.np].astype(np.complex64 if dtype == "c64" else np.complex128).astype(np.complex128)
    tol = 1e-12 if dtype == "c128" else 1e-5
    norm = m.vol_pp * np.sum(np.abs(p) ** 2, axis=0)
    assert np.allclose(n, norm, rtol=1e-12, atol=0)
    assert np.max(np.abs(d - m.vol_pp * np.sum(np.abs(p) ** 2 * r[:, None], axis=0))) <= 1e-12 * np.max(norm) * 4
    eref = m.vol_pp * np.sum((p.conj() * hx).real, axis=0)
    assert np.max(np.abs(e - eref)) <= tol * np.max(np.abs(eref))


@pytest.mark.parametrize("dtype,nst", [("c128", 5), ("c64", 18)])
@pytest.mark.parametrize("zb", [0, 4])
def test_bloch_phases(cuda, dtype, nst, zb, monkeypatch):
    import torch
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh((18, 16, 7), 0.3, periodic=True)
    psi = _states(m, nst, 9)
    k = np.array([0.4, -0.3, 0.9])
    pc = np.exp(1j * ((m.x[m.np:] - m.x[m.per_inner]) @ k))
    var, s = TMEM[dtype]
    monkeypatch.setenv(var, s.format(zb=zb))
    H = _ham(m)
    H.set_phase_corr(pc)
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    x = torch.from_numpy(psi).to(cuda).to(tdt)
    y = torch.full((m.np, nst), float("nan"), dtype=tdt, device=cuda)
    H.apply(x, y)
    ref = _oracle(m, bc="periodic", phase_corr=pc).apply(psi)
    assert rel_maxnorm_per_state(y.cpu().numpy(), ref) <= TOL[dtype]
    assert H.status() == 0


@pytest.mark.parametrize("phases", [False, True])
@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_group_of_unequal_spacings_and_phases(cuda, dtype, phases):
    import torch
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    hams, xs = [], []
    for i, (n, h, nst) in enumerate([(12, 0.25, 3), (17, 0.3, 9), (20, 0.3, 4)]):
        m = index_box_mesh((n, n + 1, n - 3), h, periodic=phases)
        H = _ham(m, v=np.random.default_rng(i).uniform(-1, 0, m.np))
        if phases:
            H.set_phase_corr(np.exp(1j * ((m.x[m.np:] - m.x[m.per_inner]) @ np.array([0.2, 0.1, -0.3]))))
        hams.append(H)
        ld = nst + (nst % 2)
        x = torch.zeros((m.np_part, ld), dtype=tdt, device=cuda)
        x[:, :nst] = torch.from_numpy(_states(m, nst, 20 + i)).to(cuda).to(tdt)
        xs.append(x)
    single = [x.clone() for x in xs]
    for H, x in zip(hams, single):
        for _ in range(2):
            H.taylor_step(x, 0.004)
    for graph in (False, True):
        ys = [x.clone() for x in xs]
        lib.Group(hams).taylor_steps(ys, 2, 0.004, graph=graph)
        for y, x in zip(ys, single):
            assert (y - x).abs().max().item() <= (1e-14 if dtype == "c128" else 1e-6) * x.abs().max().item()


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("nst", [2, 8, 10, 16, 18, 32, 34, 66])
@pytest.mark.parametrize("phased", [False, True])
@pytest.mark.parametrize("spheres", ["few", "many projectors", "many spheres"])
def test_ket_widths(cuda, dtype, nst, phased, spheres):
    """Overlapping spheres of unequal projector counts: three (rows of one to three
    matrices in well-filled blocks), three with 18 projectors on average whose points
    come in any order, and forty small ones (lists of a few rows each: one row at a time at every width)."""
    import torch
    from hpsi.mesh import sphere_mesh
    rng = np.random.default_rng(31)
    m = sphere_mesh(3.0, 0.3)
    x = m.x[: m.np]
    atoms = [((0.0, 0.1, 0.2), 1.3, 9), ((0.9, 0.0, 0.0), 1.2, 4), ((0.3, 0.8, 0.1), 1.0, 1)]
    if spheres == "many projectors":
        atoms = [(c, r, q + 14) for c, r, q in atoms]
    if spheres == "many spheres":
        atoms = [(rng.uniform(-1.4, 1.4, 3), 0.9, 1 + i % 9) for i in range(40)]

    class P:
        maps, mats, scals = [], [], []
    P.maps, P.mats, P.scals = [], [], []
    for c, r, q in atoms:
        sel = np.nonzero(np.sum((x - np.array(c)) ** 2, axis=1) <= r * r)[0].astype(np.int32)
        if spheres == "many projectors":  # any order of the points, some of them twice
            sel = rng.permutation(np.concatenate([sel, sel[:5]]))
        P.maps.append(sel)
        P.mats.append(rng.standard_normal((len(sel), q)))
        P.scals.append(rng.uniform(-1, 1, q) * m.vol_pp)
    H = _ham(m, proj=P)
    ph = [np.exp(1j * rng.uniform(0, 6, len(s))) if phased else np.ones(len(s)) for s in P.maps]
    if phased:
        H.set_projector_phases(ph)
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    psi = _states(m, nst, 33)
    xt = torch.from_numpy(psi).to(cuda).to(tdt)
    proj = torch.zeros((H.nprojections(), nst), dtype=tdt, device=cuda)
    H.projector_bra(xt, proj)
    bra = np.concatenate([np.asarray(s)[:, None] * (mt.T @ (psi[mp] * f[:, None]))
                          for mp, mt, s, f in zip(P.maps, P.mats, P.scals, ph)])
    tol = 1e-12 if dtype == "c128" else 2e-5
    assert np.max(np.abs(proj.cpu().numpy() - bra)) <= tol * np.max(np.abs(bra))
    out = xt[: m.np].clone()
    H.projector_ket(proj, out, a=0.5 - 0.25j)
    ref = psi[: m.np].copy()
    off = 0
    for mp, mt, f in zip(P.maps, P.mats, ph):
        np.add.at(ref, mp, (0.5 - 0.25j) * (mt @ bra[off: off + mt.shape[1]]) * np.conj(f)[:, None])
        off += mt.shape[1]
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= tol * np.max(np.abs(ref))
