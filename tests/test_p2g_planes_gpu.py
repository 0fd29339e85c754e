"""P2G with four lanes per cell and a plane of cells at a time: uneven cells.

Cells of one warp hold 0 to 70 particles, planes and whole tiles are empty, and
one particle's velocity is infinite: it may spoil only the nodes that its own
stencil reaches.  Both spacings: 1/h a power of two (a multiplication) and not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 9, 8), (3, 20, 17)])
@pytest.mark.parametrize("h", [1.0 / 16, 0.07])
@pytest.mark.parametrize("bad", [0.0, np.inf])
def test_uneven_cells_match_oracle(oracle, gpu, dims, h, bad):
    import torch as t

    from simcraft_b200 import fluid
    rng = np.random.default_rng(41)
    count = rng.choice([0, 0, 1, 2, 33, 70], size=dims)
    count[:, dims[1] // 2, :] = 0
    count[dims[0] // 2] = 0
    count[:, :, 0] = 0
    cells = np.repeat(np.argwhere(np.ones(dims, bool)), count.ravel(), axis=0)
    pos = (cells + rng.uniform(0.02, 0.98, cells.shape)) * h
    vel = rng.uniform(-1, 1, pos.shape)
    if bad:
        vel[len(vel) // 3] = bad
    order = rng.permutation(len(pos))
    pos, vel = np.ascontiguousarray(pos[order]), np.ascontiguousarray(vel[order])
    with np.errstate(all="ignore"):
        ref = oracle.p2g(pos, vel, dims, h, flip=True)
    got = {k: a.cpu().numpy() for k, a in
           fluid.p2g(t.from_numpy(pos).cuda(), t.from_numpy(vel).cuda(), dims, h, flip=True).items()}
    # at most 64 cells' 70 particles meet in a node: n eps = 4480 * 1.1e-16 = 5e-13 of the sum of
    # the terms' magnitudes, twice (two orders), and |v| <= 1
    for g in "uvw":
        np.testing.assert_array_equal(got[g + "valid"], ref[g + "valid"])
        np.testing.assert_allclose(got[g + "w"], ref[g + "w"], rtol=1e-12, atol=1e-15)
        fin = np.isfinite(ref[g])
        np.testing.assert_array_equal(np.isfinite(got[g]), fin)
        np.testing.assert_allclose(got[g][fin], ref[g][fin], rtol=0, atol=3e-12)
