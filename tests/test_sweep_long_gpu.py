"""Sweeps of long thin grids: more than 4096 tiles along x or y."""
import numpy as np
import pytest

from helpers import rel_l2
from test_sweep_rings_gpu import _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,solve", [((65552, 3, 2), True), ((66000, 17, 1), False), ((5, 33000, 2), True),
                                        ((40, 32800, 1), False)])
def test_precond_and_solves_of_long_grids(oracle, gpu, dims, solve):
    import torch
    from simcraft_b200.solver import CRIT_REL_L2, PREC_FP64, PREC_MIXED, CgSolver3D

    adiag, an, act = _system(dims, False, 8)
    r = np.random.default_rng(9).uniform(-1, 1, dims) * act
    s = CgSolver3D(*dims)
    s.upload(adiag, an, r, act)
    z = torch.zeros(dims, dtype=torch.float64, device="cuda")
    s.precond(torch.from_numpy(r).cuda(), z)
    # 1e-12: the bound the preconditioner has against the oracle at every other size
    assert rel_l2(z.cpu().numpy(), oracle.mic_precond(adiag, an, r, act), act.astype(bool)) < 1e-12
    for precision in (PREC_FP64, PREC_MIXED) if solve else ():
        s = CgSolver3D(*dims, tol=1e-10, max_iter=500, criterion=CRIT_REL_L2, precision=precision)
        p = np.zeros(dims)
        s.solve(adiag, an, r, act, p)
        assert s.last_stats["true_rel_l2"] < 2e-10
