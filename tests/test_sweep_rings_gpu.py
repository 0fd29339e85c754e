"""The sweeps' boundary rings over many turns: a ring entry gets its next value only when
the last one is taken, in the block, in the cluster and across mailboxes.

Long columns (a ring of 8 entries turns dozens of times a tile), cluster shapes from one
block to 4 x 4, blocks that go through several tiles, bands of tiles without an active
cell so that a block skips tiles between swept ones, and single columns.  Every repeat
gives the same bits, and the preconditioner is the oracle's."""
import numpy as np
import pytest

from helpers import rel_l2

pytestmark = pytest.mark.gpu


def _system(dims, bands, seed):
    """A symmetric seven-point system with couplings in (-1, 0) between active cells."""
    rng = np.random.default_rng(seed)
    act = rng.uniform(0, 1, dims) < 0.95
    if bands:  # whole 16-column and 8-row tiles without fluid
        act[32:48] = False
        act[:, 24:32] = False
    an = [np.zeros(dims) for _ in range(6)]
    adiag = rng.uniform(0.1, 0.3, dims)
    for axis, (low, up) in enumerate(((0, 1), (3, 2), (5, 4))):
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[axis], hi[axis] = slice(0, -1), slice(1, None)
        lo, hi = tuple(lo), tuple(hi)
        c = -rng.uniform(0.2, 1.0, act[lo].shape) * (act[lo] & act[hi])
        an[low][hi] = c
        an[up][lo] = c
        adiag[lo] -= c
        adiag[hi] -= c
    return np.where(act, adiag, 0.0), an, np.ascontiguousarray(act.astype(np.uint8))


CASES = [((1, 1, 1), False), ((1, 1, 37), False), ((16, 8, 400), False), ((16, 32, 301), False), ((48, 8, 203), False),
         ((64, 64, 260), False), ((64, 64, 130), True), ((150, 130, 90), True), ((256, 256, 67), False),
         ((300, 200, 41), True)]


@pytest.mark.parametrize("dims,bands", CASES)
def test_precond_is_the_oracles_and_repeats(oracle, gpu, dims, bands):
    import torch
    from simcraft_b200.solver import CgSolver3D

    adiag, an, act = _system(dims, bands, 3)
    r = np.random.default_rng(4).uniform(-1, 1, dims) * act
    s = CgSolver3D(*dims)
    s.upload(adiag, an, r, act)
    rd = torch.from_numpy(r).cuda()
    z = torch.full(dims, float("nan"), dtype=torch.float64, device="cuda")
    s.precond(rd, z)
    first = z.clone()
    for _ in range(20):
        s.precond(rd, z)
        assert torch.equal(z, first)
    ref = oracle.mic_precond(adiag, an, r, act)
    # 1e-12: the bound the preconditioner has against the oracle at every other size
    if act.any():
        assert rel_l2(first.cpu().numpy(), ref, act.astype(bool)) < 1e-12


@pytest.mark.parametrize("dims,bands", [((16, 32, 301), False), ((64, 64, 130), True), ((256, 256, 67), False)])
def test_mixed_solve_repeats(oracle, gpu, dims, bands):
    from simcraft_b200.solver import CRIT_REL_L2, PREC_MIXED, CgSolver3D

    adiag, an, act = _system(dims, bands, 5)
    b = np.random.default_rng(6).uniform(-1, 1, dims) * act
    # the systems are dominated by their diagonal, which has a margin of 0.1 over row sums of
    # up to 6: a condition number below 130
    s = CgSolver3D(*dims, tol=1e-10, max_iter=500, criterion=CRIT_REL_L2, precision=PREC_MIXED)
    p = [np.zeros(dims) for _ in range(4)]
    for out in p:
        s.solve(adiag, an, b, act, out)
        assert s.last_stats["true_rel_l2"] < 2e-10
    for out in p[1:]:
        np.testing.assert_array_equal(out, p[0])
