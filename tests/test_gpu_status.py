"""The status word of a Hamiltonian's bounded waits.  No kernel is made to wait
in vain: the tests record on the host what a kernel records whose wait gave up."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 5


def _record_timeout(H):
    from hpsi import lib
    fn = lib.load().hpsi_test_record_timeout
    fn.restype, fn.argtypes = C.c_int32, [C.c_void_p]
    assert fn(H.handle) == 0


def _mesh():
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh((9, 8, 7), 0.3)
    return m, lib.DeviceMesh(m)


def _ham(m, dm):
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    return lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points())


def test_every_hamiltonian_has_its_own_word(cuda):
    m, dm = _mesh()
    hams = [_ham(m, dm) for _ in range(600)]  # more than two blocks of words
    _record_timeout(hams[0])
    _record_timeout(hams[300])
    assert [i for i, H in enumerate(hams) if H.status() == TIMEOUT] == [0, 300]
    assert all(H.status() == 0 for H in hams)  # reading clears


def test_a_word_is_not_inherited(cuda):
    m, dm = _mesh()
    for _ in range(300):
        H = _ham(m, dm)
        assert H.status() == 0
        _record_timeout(H)
        H.close()


def test_a_word_outlives_its_mesh(cuda):
    import torch
    m, dm = _mesh()
    H, other = _ham(m, dm), _ham(m, dm)
    dm.close()
    for _ in range(8):  # memory given back with the mesh would be handed out here
        torch.full((1 << 18,), 7, dtype=torch.int32, device=cuda)
        _mesh()[1].close()
    assert H.status() == 0
    _record_timeout(H)
    assert other.status() == 0 and H.status() == TIMEOUT


def test_calls_that_wait_for_the_device_report_a_timeout(cuda):
    """Every call that brings results to the host answers with the timeout as long as
    the word is set, and works again once it has been read."""
    import torch
    from hpsi import lib
    m, dm = _mesh()
    H = _ham(m, dm)
    rng = np.random.default_rng(3)
    host = np.zeros((m.np_part, 4), dtype=np.complex128)
    host[: m.np] = rng.standard_normal((m.np, 4)) + 1j * rng.standard_normal((m.np, 4))
    wide = np.zeros((m.np_part, 16), dtype=np.complex128)  # (two slabs of the host pipeline)
    x = torch.from_numpy(host).to(cuda)
    dm.orthonormalize_cholesky(x)
    eps = np.linspace(0.0, 0.01, 3)
    calls = {
        "host batch": lambda: H.apply(host, np.zeros((m.np, 4), dtype=np.complex128)),
        "host batch in slabs": lambda: H.apply(wide, np.zeros((m.np, 16), dtype=np.complex128)),
        "host step": lambda: H.taylor_step(host.copy(), 1e-3),
        "observables": lambda: H.taylor_step(x.clone(), 1e-3, observables=True),
        "propagation": lambda: H.td_propagate(x.clone(), 2, 1e-3),
        "propagation, no graph": lambda: H.td_propagate(x.clone(), 2, 1e-3, graph=False),
        "etrs": lambda: H.td_propagate(x.clone(), 2, 1e-3, propagator="etrs"),
        "lanczos": lambda: H.lanczos_step(x.clone(), 1e-3),
        "adjoint": lambda: H.adjoint_gradient(x, x.clone(), eps, 1e-3),
        "adjoint step": lambda: H.adjoint_step(x.clone(), x, 0.01, 1e-3),
        "autotune": lambda: H.autotune(ld=4),
    }
    for name, call in calls.items():
        call()
        _record_timeout(H)
        with pytest.raises(lib.HpsiError) as e:
            call()
        assert e.value.status == TIMEOUT, name
        assert H.status() == TIMEOUT, name
        call()
    assert H.status() == 0
