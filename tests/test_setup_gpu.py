"""The set-up of a system: which entries the pivots read.  A coupling to an inactive cell
enters the pivots of its diagonal neighbours as it is given; where it is not finite, and
in inactive rows, nothing reads it."""
import numpy as np
import pytest

from helpers import rel_l2
from test_sweep_rings_gpu import _system

pytestmark = pytest.mark.gpu

DIMS = [(33, 17, 9), (40, 24, 1), (5, 9, 70), (64, 32, 3)]


def _lower(act, axis):
    """Cells whose lower neighbour along axis is outside the grid or inactive."""
    out = np.ones(act.shape, bool)
    lo, hi = [slice(None)] * 3, [slice(None)] * 3
    lo[axis], hi[axis] = slice(0, -1), slice(1, None)
    out[tuple(hi)] = act[tuple(lo)] == 0
    return out


def _precond(dims, adiag, an, r, act):
    import torch
    from simcraft_b200.solver import CgSolver3D

    s = CgSolver3D(*dims)
    s.upload(adiag, an, r, act)
    z = torch.zeros(dims, dtype=torch.float64, device="cuda")
    s.precond(torch.from_numpy(r).cuda(), z)
    return z.cpu().numpy()


@pytest.mark.parametrize("dims", DIMS)
def test_finite_couplings_to_inactive_cells_count_as_given(oracle, gpu, dims):
    adiag, an, act = _system(dims, False, 31)
    rng = np.random.default_rng(32)
    for axis, low in enumerate((0, 3, 5)):
        m = _lower(act, axis) & (act != 0)
        an[low][m] = rng.uniform(-0.2, 0.0, m.sum())
    r = rng.uniform(-1, 1, dims) * act
    ref = oracle.mic_precond(adiag, an, r, act)
    # 1e-12: the bound the preconditioner has against the oracle at every other size
    assert rel_l2(_precond(dims, adiag, an, r, act), ref, act.astype(bool)) < 1e-12


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_entries_that_nothing_reads_may_be_non_finite(gpu, dims, bad):
    from simcraft_b200.solver import CRIT_REL_L2, PREC_FP64, PREC_MIXED, CgSolver3D

    adiag, an, act = _system(dims, False, 33)
    r = np.random.default_rng(34).uniform(-1, 1, dims) * act
    adiag2, an2 = adiag.copy(), [a.copy() for a in an]
    for axis, low in enumerate((0, 3, 5)):
        an2[low][_lower(act, axis) | (act == 0)] = bad
    adiag2[act == 0] = bad
    np.testing.assert_array_equal(_precond(dims, adiag2, an2, r, act), _precond(dims, adiag, an, r, act))
    for precision in (PREC_FP64, PREC_MIXED):
        p = []
        for A, N in ((adiag, an), (adiag2, an2)):
            s = CgSolver3D(*dims, tol=1e-9, max_iter=300, criterion=CRIT_REL_L2, precision=precision)
            p.append(np.zeros(dims))
            s.solve(A, N, r, act, p[-1])
            assert s.last_stats["true_rel_l2"] < 2e-9
        np.testing.assert_array_equal(p[1], p[0])
