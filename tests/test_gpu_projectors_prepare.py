"""hpsi_hamiltonian_set_projectors: the tables of the KB ket from any list of spheres."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _P:
    def __init__(self, maps, mats, scals):
        self.maps, self.mats, self.scals = maps, mats, scals


def _ket(m, dm, P, nst, cuda, phases=None):
    """H psi of the projectors alone, and its restatement in numpy."""
    import torch
    from hpsi import lib
    from hpsi.stencil import laplacian_weights, star_points
    H = lib.Hamiltonian(dm, laplacian_weights(m.spacing), star_points(), projectors=P)
    rng = np.random.default_rng(2)
    proj = rng.standard_normal((H.nprojections(), nst)) + 1j * rng.standard_normal((H.nprojections(), nst))
    out = torch.zeros((m.np, nst), dtype=torch.complex128, device=cuda)
    H.projector_ket(torch.from_numpy(proj).to(cuda), out)
    ref = np.zeros((m.np, nst), dtype=np.complex128)
    off = 0
    for mp, mt in zip(P.maps, P.mats):
        np.add.at(ref, mp, mt @ proj[off: off + mt.shape[1]])
        off += mt.shape[1]
    return out.cpu().numpy(), ref


def _spheres(case, m, rng):
    one = lambda sel, q: (np.asarray(sel, dtype=np.int32), rng.standard_normal((len(sel), q)), rng.uniform(-1, 1, q))
    if case == "the same sphere twice":
        s = rng.permutation(m.np)[:100]
        return [one(s, 3), one(s, 5)]
    if case == "an empty sphere":
        return [one([], 2), one(np.arange(40, 75), 1), one([], 1)]
    if case == "all points":
        return [one(rng.permutation(m.np), 2), one(np.arange(m.np), 1)]
    if case == "first and last row":
        return [one([m.np - 1, 0], 4)]
    if case == "a point many times":
        return [one([7] * 40 + [9], 2), one([9, 7, 9], 1)]
    # nested intervals: as many lists as spheres, the last ones of one row
    return [one(np.arange(i, 64), 1 + i % 4) for i in range(64)]


@pytest.mark.parametrize("nst", [2, 24, 48])  # both forms of the ket
@pytest.mark.parametrize("case", ["the same sphere twice", "an empty sphere", "all points", "first and last row",
                                  "a point many times", "nested"])
def test_ket_of_any_list_of_spheres(cuda, case, nst):
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    m = index_box_mesh((9, 8, 7), 0.3)
    P = _P(*zip(*_spheres(case, m, np.random.default_rng(1))))
    got, ref = _ket(m, lib.DeviceMesh(m), P, nst, cuda)
    # at most 64 + 40 projectors a point
    assert np.max(np.abs(got - ref)) <= 256 * np.finfo(float).eps * max(1.0, np.max(np.abs(ref)))


def test_a_refused_list_leaves_no_projectors(cuda):
    from hpsi import lib
    from hpsi.mesh import index_box_mesh
    from hpsi.stencil import laplacian_weights, star_points
    m = index_box_mesh((9, 8, 7), 0.3)
    H = lib.Hamiltonian(lib.DeviceMesh(m), laplacian_weights(m.spacing), star_points())
    for bad in (-1, m.np):
        H.set_projectors([np.array([1, 2])], [np.ones((2, 1))], [np.ones(1)])
        with pytest.raises(lib.HpsiError) as e:
            H.set_projectors([np.array([1, bad])], [np.ones((2, 1))], [np.ones(1)])
        assert e.value.status == 2  # HPSI_ERR_INDEX
        assert H.nprojections() == 0
