"""A resident system under changing calls: the inner method of the mixed solve switched
between two solves of the same system, the matrix applied in place, and the pressure
after a solve that failed."""
import numpy as np
import pytest

from test_sweep_rings_gpu import _system

pytestmark = pytest.mark.gpu

INNER_PCG, INNER_EISENSTAT = 0, 1


@pytest.mark.parametrize("order", [(INNER_EISENSTAT, INNER_PCG), (INNER_PCG, INNER_EISENSTAT, INNER_PCG)])
def test_the_inner_method_may_change_between_solves(gpu, order):
    from simcraft_b200.solver import CRIT_REL_L2, PREC_MIXED, CgSolver3D

    dims = (40, 24, 30)
    solver = None
    for seed in (11, 12):  # a second system in the same handle: nothing of the first may stay
        adiag, an, act = _system(dims, False, seed)
        b = np.random.default_rng(seed + 50).uniform(-1, 1, dims) * act
        opts = dict(tol=1e-10, max_iter=400, criterion=CRIT_REL_L2, precision=PREC_MIXED)
        if solver is None:
            solver = CgSolver3D(*dims, inner_method=order[0], **opts)
        solver.set_options(inner_method=order[0])
        solver.upload(adiag, an, b, act)
        for method in order:
            solver.set_options(inner_method=method)
            fresh = CgSolver3D(*dims, inner_method=method, **opts)
            fresh.upload(adiag, an, b, act)
            p = []
            for s in (fresh, solver):
                st = s.solve_resident()
                assert st["status"] == 1 and st["true_rel_l2"] < 2e-10
                p.append(s.download(np.zeros(dims)))
            np.testing.assert_array_equal(p[1], p[0])


@pytest.mark.parametrize("dims", [(1, 1, 1), (33, 17, 9), (96, 64, 80)])
@pytest.mark.parametrize("shift", [0, 1, 777, -1, -777])
def test_apply_to_overlapping_vectors(gpu, dims, shift):
    import torch
    from simcraft_b200.solver import CRIT_REL_L2, CgSolver3D

    adiag, an, act = _system(dims, False, 13)
    n = int(np.prod(dims))
    rhs = np.random.default_rng(14).uniform(-1, 1, dims) * act
    s = CgSolver3D(*dims, tol=1e-10, max_iter=400, criterion=CRIT_REL_L2)
    s.upload(adiag, an, rhs, act)
    x = torch.from_numpy(np.random.default_rng(15).uniform(-1, 1, dims)).cuda()
    ref = torch.empty_like(x)
    s.apply(x, ref)
    s.solve_resident()
    before = s.download(np.zeros(dims))
    buf = torch.zeros(n + 800, dtype=torch.float64, device="cuda")
    at = max(0, -shift)
    xv, bv = buf[at:at + n].view(dims), buf[at + shift:at + shift + n].view(dims)
    for _ in range(5):
        xv.copy_(x)
        s.apply(xv, bv)
        assert torch.equal(bv, ref)
    s.solve_resident()  # the solver's own arrays are as they were
    np.testing.assert_array_equal(s.download(np.zeros(dims)), before)


def test_after_a_failed_solve_the_pressure_is_not_the_previous_one(gpu):
    """A right-hand side with an infinite value: the solve fails at its first residual with
    p = 0, and that is what a download gives."""
    from simcraft_b200._capi import CapiError
    from simcraft_b200.solver import CRIT_REL_L2, CgSolver3D

    dims = (24, 20, 18)
    adiag, an, act = _system(dims, False, 16)
    rhs = np.random.default_rng(17).uniform(-1, 1, dims) * act
    s = CgSolver3D(*dims, tol=1e-10, max_iter=400, criterion=CRIT_REL_L2)
    s.upload(adiag, an, rhs, act)
    s.solve_resident()
    good = s.download(np.zeros(dims))
    assert np.abs(good).max() > 0.0
    bad = rhs.copy()
    bad[tuple(np.argwhere(act)[act.sum() // 2])] = np.inf
    s.upload(adiag, an, bad, act)
    with pytest.raises(CapiError):
        s.solve_resident()
    np.testing.assert_array_equal(s.download(np.full(dims, 7.0)), np.zeros(dims))
    s.upload(adiag, an, rhs, act)
    s.solve_resident()
    np.testing.assert_array_equal(s.download(np.zeros(dims)), good)
