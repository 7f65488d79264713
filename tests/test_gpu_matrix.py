"""Overlap matrix and Cholesky orthonormalisation at the edges of their tiles:
64 real lanes (32 states), 16 points or lanes per step, and the largest triangle
the shared-memory Cholesky holds (168 states)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh():
    from hpsi.mesh import index_box_mesh
    return index_box_mesh((13, 11, 9), 0.4)  # 1287 points: not a multiple of 16 or 64


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("nst,ld", [(1, 2), (5, 6), (31, 32), (32, 32), (33, 36), (64, 72), (97, 98), (168, 168), (169, 170)])
def test_overlap_and_orthonormalisation(cuda, dtype, nst, ld):
    import torch
    from hpsi import lib
    m = _mesh()
    rng = np.random.default_rng(nst)
    cdt = np.complex128 if dtype == "c128" else np.complex64
    a, b = (np.full((m.np_part, ld), np.nan, dtype=cdt) for _ in range(2))
    for x in (a, b):
        x[: m.np, :nst] = rng.standard_normal((m.np, nst)) + 1j * rng.standard_normal((m.np, nst))
    dm = lib.DeviceMesh(m)
    xa, xb = torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda)
    A, B = (x[: m.np, :nst].astype(np.complex128) for x in (a, b))
    # sums of np products of order 1 in FP64: rounding error below np * eps of
    # the sum of magnitudes (np)
    tol = 4 * m.np * np.finfo(float).eps * m.np * m.vol_pp
    S = dm.dotp_matrix(xa, xb, nst=nst)
    assert np.max(np.abs(S - m.vol_pp * (A.conj().T @ B))) <= tol
    Sa = dm.dotp_matrix(xa, xa, nst=nst)
    assert np.max(np.abs(Sa - m.vol_pp * (A.conj().T @ A))) <= tol
    assert np.array_equal(Sa, Sa.conj().T)
    dm.orthonormalize_cholesky(xa, nst=nst)
    U = np.linalg.cholesky(m.vol_pp * (A.conj().T @ A)).conj().T
    ref = np.linalg.solve(U.T, A.T).T
    got = xa.cpu().numpy()
    # the Gram matrix is well conditioned (np >> nst): a few hundred roundings
    eps = 1e-13 if dtype == "c128" else 1e-6
    assert np.max(np.abs(got[: m.np, :nst] - ref)) <= eps * np.max(np.abs(ref))
    # nothing beyond the batch is touched
    assert np.isnan(got[m.np:]).all() and np.isnan(got[:, nst:]).all()


def test_indefinite_overlap_is_refused(cuda):
    import torch
    from hpsi import lib
    m = _mesh()
    dm = lib.DeviceMesh(m)
    x = torch.zeros((m.np_part, 4), dtype=torch.complex128, device=cuda)
    x[: m.np, 0] = 1.0
    keep = x.clone()
    with pytest.raises(lib.HpsiError):
        dm.orthonormalize_cholesky(x, nst=2)  # a zero state
    assert torch.equal(x, keep)


def test_orthonormalisation_of_many_states(cuda):
    """1537 states: the triangular update has no limit of its own."""
    import torch
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh((17, 17, 17), 0.4)
    dm = lib.DeviceMesh(m)
    nst = 1537
    g = torch.Generator(device=cuda).manual_seed(7)
    x = torch.randn((m.np, nst), dtype=torch.complex128, device=cuda, generator=g)
    dm.orthonormalize_cholesky(x)
    S = dm.dotp_matrix(x, x)
    # condition of the overlap about (1.56 / 0.44)^2 = 13 (np / nst = 3.2): the
    # overlap of the result is the unit matrix to condition * nst * eps at most
    assert np.max(np.abs(S - np.eye(nst))) <= 13 * nst * np.finfo(float).eps


def test_too_many_states_are_refused(cuda):
    import torch
    from hpsi import lib
    m = _mesh()
    x = torch.zeros((m.np, 3074), dtype=torch.complex64, device=cuda)
    with pytest.raises(lib.HpsiError, match="3072"):
        lib.DeviceMesh(m).orthonormalize_cholesky(x, nst=3073)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("nst,same", [(641, True), (480, False), (512, True)])
def test_long_sums_are_folded(cuda, dtype, nst, same):
    """One split (641 states, or two batches of 480) or few over 216,000 points.  The
    first row is so large that every later product is lost when it is added to a
    plain running sum: a sum in one chain is off by 5e-12."""
    import torch
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh((60, 60, 60), 0.25)
    tdt = torch.complex128 if dtype == "c128" else torch.complex64
    ld = nst + nst % 2
    x = torch.full((m.np, ld), 0.66, dtype=tdt, device=cuda)
    x[0] = 2.0 ** 27
    small = float(x[1, 0].real.item()) ** 2
    S = lib.DeviceMesh(m).dotp_matrix(x, x if same else x.clone(), nst=nst)
    ref = m.vol_pp * (2.0 ** 54 + (m.np - 1) * small)
    # plain sums run over 8192 points at most: 8192 roundings of half an eps each
    assert np.max(np.abs(S - ref)) <= 8192 * np.finfo(float).eps / 2 * ref


@pytest.mark.parametrize("offset", [0, 1, 2])
def test_overlap_of_an_unaligned_single_state(cuda, offset):
    """FP32 batches of width 1 may start on any 4-byte boundary."""
    import ctypes as C
    import torch
    from hpsi import lib
    m = _mesh()
    dm = lib.DeviceMesh(m)
    g = torch.Generator(device=cuda).manual_seed(5)
    buf = torch.randn(2 * m.np + 4, device=cuda, generator=g)
    b = lib.Batch()
    b.dtype, b.ptr, b.ld, b.npts, b.nst = lib.HPSI_C64, buf.data_ptr() + 4 * offset, 1, m.np, 1
    out = np.zeros(2)
    lib.check(lib.load().hpsi_dotp_matrix(dm.handle, C.byref(b), C.byref(b), out.ctypes.data_as(C.POINTER(C.c_double)),
                                          None))
    x = buf[offset: offset + 2 * m.np].double().cpu().numpy()
    torch.cuda.synchronize()
    ref = m.vol_pp * float(x @ x)
    assert abs(out[0] - ref) <= 4 * m.np * np.finfo(float).eps * ref and out[1] == 0.0
