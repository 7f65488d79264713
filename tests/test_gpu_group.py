"""Grouped systems (one persistent launch per pass) and the autotuner."""
import numpy as np
import pytest

from helpers import rel_maxnorm_per_state

pytestmark = pytest.mark.gpu


def _system(seed, n, nst, natoms):
    from hpsi import fixtures
    from hpsi.mesh import index_box_mesh
    rng = np.random.default_rng(seed)
    m = index_box_mesh((n, n + 1, n - 1), 0.25)
    v = fixtures.soft_coulomb(m, rng)
    proj = fixtures.kb_projectors(m, natoms, rng, radius=0.8, min_dist=0.6, place_radius=0.8) if natoms else None
    psi = fixtures.random_states(m, nst, rng)
    return m, v, proj, psi


def test_group_matches_single_systems(cuda):
    import torch
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    specs = [(1, 12, 4, 2), (2, 17, 7, 0), (3, 9, 16, 3), (4, 21, 5, 1), (5, 14, 12, 2)]
    hams, xs, refs = [], [], []
    for seed, n, nst, natoms in specs:
        m, v, proj, psi = _system(seed, n, nst, natoms)
        dm = lib.DeviceMesh(m)
        ham = lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points(), v=v, projectors=proj)
        ld = 1 << (nst - 1).bit_length()
        x = torch.zeros((m.np_part, ld), dtype=torch.complex128, device=cuda)
        x[:, :nst] = torch.from_numpy(psi)
        r = x.clone()
        for _ in range(3):
            ham.taylor_step(r, 0.02, nst=nst)
        hams.append((dm, ham))
        xs.append(x)
        refs.append(r)
    g = lib.Group([h for _, h in hams])
    for graph in (False, True):
        ys = [x.clone() for x in xs]
        g.taylor_steps(ys, 3, 0.02, graph=graph)
        torch.cuda.synchronize()
        for y, r, (seed, n, nst, natoms) in zip(ys, refs, specs):
            np_ = r.shape[0]
            assert rel_maxnorm_per_state(y.cpu().numpy()[:, :nst], r.cpu().numpy()[:, :nst]) <= 1e-14
    g.close()


def test_autotune_keeps_results(cuda):
    import torch
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    m, v, proj, psi = _system(7, 20, 8, 2)
    dm = lib.DeviceMesh(m)
    ham = lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points(), v=v, projectors=proj)
    x = torch.from_numpy(psi).to(cuda)
    y0 = torch.zeros((m.np, 8), dtype=torch.complex128, device=cuda)
    ham.apply(x, y0)
    shape, ms = ham.autotune(lib.HPSI_C128, 8)
    assert shape["sc"] in (1, 2, 4, 8) and ms > 0
    y1 = torch.zeros_like(y0)
    ham.apply(x, y1)
    assert rel_maxnorm_per_state(y1.cpu().numpy(), y0.cpu().numpy()) <= 1e-14
    x32 = x.to(torch.complex64)
    shape32, _ = ham.autotune(lib.HPSI_C64, 8)
    assert shape32["sc"] in (2, 4, 8)


# shape overrides of the grouped launch: the blocked pass, the tensor-memory pass with
# z blocks of five planes
FORMS = {"default": None,
         "blocked": {"c128": "8,2,0,9,1,2,0,8", "c64": "16,2,0,9,1,2,1,8"},
         "tensor memory": {"c128": "8,2,5,9,1,2,0,8,0,0,0,1", "c64": "16,2,5,9,1,2,1,8,0,0,0,1"}}


def _force(monkeypatch, form, dtype):
    if FORMS[form]:
        monkeypatch.setenv({"c128": "HPSI_PASS_SHAPE64", "c64": "HPSI_PASS_SHAPE32"}[dtype], FORMS[form][dtype])


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_group_blocked_pass_matches_single_systems(cuda, dtype, form, monkeypatch):
    """Every width a multiple of the blocked pass's chunk (8 complex128 / 16
    complex64 states): the grouped launch of each form (without a field: the blocked
    pass in its field-free form) against single systems in the default one."""
    import torch
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    chunk = 8 if dtype == "c128" else 16
    specs = [(11, 13, 5, 2), (12, 18, chunk + 3, 0), (13, 10, 2 * chunk, 3), (14, 22, 3, 1)]
    hams, xs, refs, nsts = [], [], [], []
    for seed, n, nst, natoms in specs:
        m, v, proj, psi = _system(seed, n, nst, natoms)
        dm = lib.DeviceMesh(m)
        ham = lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points(), v=v, projectors=proj)
        ld = chunk * ((nst + chunk - 1) // chunk)
        x = torch.zeros((m.np_part, ld), dtype=tdt, device=cuda)
        x[:, :nst] = torch.from_numpy(psi).to(tdt)
        r = x.clone()
        for _ in range(3):
            ham.taylor_step(r, 0.02)
        hams.append((dm, ham))
        xs.append(x)
        refs.append(r)
        nsts.append(nst)
    _force(monkeypatch, form, dtype)
    g = lib.Group([h for _, h in hams])
    tol = 1e-13 if dtype == "c128" else 1e-6
    for graph in (False, True):
        ys = [x.clone() for x in xs]
        g.taylor_steps(ys, 3, 0.02, graph=graph)
        torch.cuda.synchronize()
        for y, r, nst in zip(ys, refs, nsts):
            a = y.cpu().numpy()[:, :nst].astype(np.complex128)
            b = r.cpu().numpy()[:, :nst].astype(np.complex128)
            assert rel_maxnorm_per_state(a, b) <= tol
    g.close()


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_group_with_laser_field_matches_single_systems(cuda, dtype, form, monkeypatch):
    """Systems with a laser field in the group (the blocked pass with the field
    term): each system as its own Taylor steps with the same field."""
    import torch
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    chunk = 8 if dtype == "c128" else 16
    specs = [(21, 14, chunk, 2), (22, 17, 2 * chunk, 0), (23, 11, chunk, 1)]
    fields = [((0.3, -0.5, 0.8), 0.05), None, ((0.0, 0.0, 1.0), -0.02)]
    hams, xs, refs = [], [], []
    for (seed, n, nst, natoms), fld in zip(specs, fields):
        m, v, proj, psi = _system(seed, n, nst, natoms)
        dm = lib.DeviceMesh(m)
        ham = lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points(), v=v, projectors=proj)
        if fld is not None:
            ham.set_field(*fld)
        x = torch.zeros((m.np_part, nst), dtype=tdt, device=cuda)
        x[:, :nst] = torch.from_numpy(psi).to(tdt)
        r = x.clone()
        for _ in range(3):
            ham.taylor_step(r, 0.02)
        hams.append((dm, ham))
        xs.append(x)
        refs.append(r)
    _force(monkeypatch, form, dtype)
    g = lib.Group([h for _, h in hams])
    tol = 1e-13 if dtype == "c128" else 1e-6
    ys = [x.clone() for x in xs]
    g.taylor_steps(ys, 3, 0.02)
    torch.cuda.synchronize()
    for y, r in zip(ys, refs):
        a = y.cpu().numpy().astype(np.complex128)
        b = r.cpu().numpy().astype(np.complex128)
        assert rel_maxnorm_per_state(a, b) <= tol
    g.close()


@pytest.mark.parametrize("dtype,widths", [("c128", (1, 2, 1)), ("c128", (2, 2, 2)), ("c128", (1, 3, 2)),
                                          ("c64", (2, 4, 2)), ("c64", (4, 4, 4)), ("c64", (2, 6, 4))])
def test_group_of_narrow_batches(cuda, dtype, widths):
    """More than 500,000 points in all: batches of at most a quarter of the chunk in the
    one-complex pass, with one wider batch among them in the tensor-memory pass."""
    import torch
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    from hpsi.stencil import laplacian_weights, star_points
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    gen = torch.Generator(device=cuda).manual_seed(4)
    hams, xs = [], []
    for i, ld in enumerate(widths):
        m = index_box_mesh((56, 57 + i, 55), 0.3)
        v = np.random.default_rng(i).uniform(-1, 0, m.np)
        hams.append(lib.Hamiltonian(lib.DeviceMesh(m), laplacian_weights(m.spacing), star_points(), v=v))
        xs.append(torch.randn((m.np_part, ld), dtype=tdt, device=cuda, generator=gen))
    single = [x.clone() for x in xs]
    for H, x in zip(hams, single):
        for _ in range(2):
            H.taylor_step(x, 0.004)
    ys = [x.clone() for x in xs]
    lib.Group(hams).taylor_steps(ys, 2, 0.004)
    for H, y, x in zip(hams, ys, single):
        n = H.dmesh.mesh.np
        assert (y - x)[:n].abs().max().item() <= (1e-13 if dtype == "c128" else 1e-6) * x[:n].abs().max().item()


def test_autotune_of_one_state_knows_the_one_complex_pass(cuda):
    """One state on a large mesh: the one-complex pass (2 rows per thread) takes 2/3 of
    the tensor-memory pass's time, which the autotuner must not choose instead."""
    import torch
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    from hpsi.stencil import laplacian_weights, star_points
    m = index_box_mesh((96, 96, 96), 0.25)
    H = lib.Hamiltonian(lib.DeviceMesh(m), laplacian_weights(m.spacing), star_points())
    x = torch.randn((m.np_part, 1), dtype=torch.complex128, device=cuda)
    y0, y1 = (torch.zeros((m.np, 1), dtype=torch.complex128, device=cuda) for _ in range(2))
    H.apply(x, y0)
    shape, _ = H.autotune(lib.HPSI_C128, 1)
    assert shape["ry"] == 2 and shape["sc"] == 1
    H.apply(x, y1)
    assert (y1 - y0).abs().max().item() <= 1e-13 * y0.abs().max().item()
