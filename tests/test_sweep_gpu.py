"""The wavefront sweeps (sc_sweep.cuh) where their decomposition can go wrong: one
column up to several tiles per block, remainders in x, y and z of the 16 x 8 column
tiles, their 8 x 4 warp tiles and the chunks of four steps, tiles shorter than the
stages a block keeps in flight (more tiles than blocks, so that a block goes from
tile to tile), cluster shapes along x, along y and square, tiles without an active
cell between active ones.  The preconditioner against the oracle, the solves against
the oracle's solution; a second application is the same bit for bit."""
import numpy as np
import pytest

from helpers import poisson_system, rel_l2

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1), (8, 4, 1), (9, 5, 2), (17, 9, 3), (16, 8, 13), (15, 7, 22), (40, 8, 54), (16, 70, 33), (33, 17, 6),
        (64, 64, 5), (130, 70, 9), (320, 144, 2), (200, 168, 7)]


def _system(oracle, dims, fill=0.5):
    S = poisson_system(oracle, 0, dims=dims, seed=11, fill=fill)
    if not S["active"].any():
        pytest.skip("no active cell")
    return S


@pytest.mark.parametrize("dims", DIMS)
def test_precond_at_the_edges_of_the_decomposition(oracle, gpu, dims):
    import torch
    from simcraft_b200.solver import CgSolver3D

    S = _system(oracle, dims, fill=0.7)
    s = CgSolver3D(*dims)
    s.upload(S["adiag"], S["an"], S["rhs"], S["active"])
    r = np.random.default_rng(5).uniform(-1, 1, dims)
    z = [torch.full(dims, float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    for out in z:
        s.precond(torch.from_numpy(r).cuda(), out)
    assert torch.equal(z[0], z[1])
    a = S["active"].astype(bool)
    ref = oracle.mic_precond(S["adiag"], S["an"], r, S["active"])
    # 1e-12: the bound the preconditioner has against the oracle at every other size
    assert rel_l2(z[0].cpu().numpy(), ref, a) < 1e-12


@pytest.mark.parametrize("dims", [(17, 9, 3), (70, 16, 33), (130, 70, 9), (320, 144, 2), (200, 168, 7)])
@pytest.mark.parametrize("mixed", [False, True])
def test_solve_at_the_edges_of_the_decomposition(oracle, gpu, dims, mixed):
    from simcraft_b200.solver import CRIT_REL_L2, PREC_FP64, PREC_MIXED, CgSolver3D

    S = _system(oracle, dims, fill=0.3)
    s = CgSolver3D(*dims, tol=1e-10, max_iter=2000, criterion=CRIT_REL_L2, precision=PREC_MIXED if mixed else PREC_FP64)
    p = [np.zeros(dims) for _ in range(2)]
    for out in p:
        s.solve(S["adiag"], S["an"], S["rhs"], S["active"], out)
    assert s.last_stats["true_rel_l2"] < 2e-10
    np.testing.assert_array_equal(p[0], p[1])
    ref, _, _ = oracle.pcg_solve(S["adiag"], S["an"], S["rhs"], S["active"], tol=1e-12, max_iter=5000,
                                 criterion=oracle.CRIT_REL_L2)
    a = S["active"].astype(bool)
    # a relative residual of 1e-10 times the condition number of these systems (below 1e5)
    assert rel_l2(p[0], ref, a) < 1e-5
