"""The surface export where its blocks of 4096 cubes and lists of crossing cubes can go
wrong: cube counts just below, at and above a block, rows longer than a block's 256
lanes and rows of a few cubes, columns and planes, and noise, where nearly every cube
crosses and a block's lists are at their fullest.  Bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx + 1)(ny + 1)(nz + 1) cubes
DIMS = [(1, 1, 1), (15, 15, 15), (15, 15, 14), (15, 16, 15), (1, 1, 2047), (1, 1, 2048), (2, 1, 700), (3, 900, 1), (1200, 2, 2),
        (31, 31, 31), (17, 40, 31), (5, 6, 300)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("kind", ["noise", "plane"])
def test_mesh_at_the_edges_of_the_blocks(oracle, gpu, dims, kind):
    import torch
    from simcraft_b200.surface import rebuild_surface

    rng = np.random.default_rng(sum(dims))
    if kind == "noise":
        sdf = rng.uniform(-1, 1, dims)
    else:
        x, y, z = np.meshgrid(*(np.arange(n, dtype=float) for n in dims), indexing="ij")
        sdf = x / dims[0] + y / dims[1] + z / dims[2] - 1.3 + 0.01 * rng.uniform(-1, 1, dims)
    sp = (0.7, 1.1, 0.9)
    ref = oracle.rebuild_surface(sdf, sp)
    V, N, I = (a.cpu().numpy() for a in rebuild_surface(torch.from_numpy(sdf).cuda(), sp))
    np.testing.assert_array_equal(V, ref[0])
    np.testing.assert_array_equal(N, ref[1])
    np.testing.assert_array_equal(I.astype(np.int64), ref[2].astype(np.int64))
