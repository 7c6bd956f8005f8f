"""Floodfill tiles with more runs than the label writer stages in shared
memory, in rows that are and are not whole words, and arrays off the 16-byte
grid, against the oracle's floodfill."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh

pytestmark = pytest.mark.gpu

SHAPES = [(1, 150, 250, 3), (1, 150, 256, 3), (2, 129, 225, 2), (1, 3, 33000, 2), (1, 40, 31, 5)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("p", [0.3, 0.55])
def test_noise_labels(oracle, dev, shape, p):
    g = np.random.default_rng(sum(shape)).random(shape) < p
    assert np.array_equal(cubvh.floodfill(torch.from_numpy(g).to(dev)).cpu().numpy(), oracle.floodfill(g))
    off = torch.empty(g.size + 1, dtype=torch.bool, device=dev)[1:].view(shape)   # an odd address
    off.copy_(torch.from_numpy(g))
    assert np.array_equal(cubvh.floodfill(off).cpu().numpy(), oracle.floodfill(g))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("first", [0.0, 1.0])
def test_noise_signs(oracle, dev, shape, first):
    """first: the volume's first voxel is occupied or free."""
    rng = np.random.default_rng(sum(shape) + 1)
    u = rng.random(shape).astype(np.float32)
    u[rng.random(shape) < 0.4] = 0.0
    u[:, 0, 0, 0] = first
    u.reshape(-1)[rng.choice(u.size, 5, replace=False)] = np.nan
    eps = np.float32(0.05)
    lab = oracle.floodfill(u < eps)
    want = u - eps
    flip = (lab != lab[:, :1, :1, :1]) & (want > 0)
    want[flip] = -want[flip]
    for shift in (0, 1):
        t = torch.empty(u.size + shift, device=dev)[shift:].view(shape)
        t.copy_(torch.from_numpy(u))
        got = cubvh.udf_to_sdf(t, eps=float(eps)).cpu().numpy()
        assert np.array_equal(got, want, equal_nan=True)
