"""Floodfill of grids of very many small slices, whose components are chains of
one root per slice: the kernel that shortens the chains, and what they cost."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 16, 16, 4096), (2, 3, 5, 1024), (1, 5, 7, 1023), (1, 1, 1, 3000), (1, 40, 33, 1025)])
@pytest.mark.parametrize("kind", ["free", "columns", "noise", "plugs"])
def test_deep(oracle, dev, shape, kind):
    """One column, a column per second x, branching ones, and columns cut in four (B slices of D each in a row)."""
    rng = np.random.default_rng(sum(shape))
    g = np.zeros(shape, bool)
    m = g.reshape(shape[0], shape[3], shape[2], shape[1])     # the order of the voxels in memory: z, y, x
    if kind == "columns":
        m[..., 1::2] = True
    elif kind == "noise":
        m[:] = rng.random(m.shape) < 0.3
    elif kind == "plugs":
        m[:, ::max(1, shape[3] // 4)] = True
    t = torch.from_numpy(g).to(dev)
    assert np.array_equal(cubvh.floodfill(t).cpu().numpy(), oracle.floodfill(g))


def test_deep_cost(dev):
    """A free column of 4,096 slices costs about as much as a free grid of as many voxels; 20 times with chains
    walked to their end."""
    def ms(shape):
        grid = torch.zeros(shape, dtype=torch.bool, device=dev)
        t = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            cubvh.floodfill(grid)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t)

    assert ms((1, 16, 16, 4096)) < 6 * ms((1, 128, 128, 64))
