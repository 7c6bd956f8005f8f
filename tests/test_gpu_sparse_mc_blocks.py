"""Sparse marching cubes at the edges of its blocks and key types.

The count and emit kernels prefix their counts per block of 256 voxels, the
merge kernels their run starts per block of 256 vertices, and the edge keys
are 32-bit where (rx * ry * rz * 3) fits in 32 bits, 64-bit otherwise (rx, ry,
rz: corners along each axis).  Vertices and triangles must equal the oracle's
restatement bit for bit."""

import os

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh

HERE = os.path.dirname(os.path.abspath(__file__))
TABLE = np.load(os.path.join(HERE, "golden", "ref_mc_cases.npz"))["tri_edges"]


def _voxels(n, corners_per_axis, seed):
    """n voxels whose corner range is exactly corners_per_axis along each axis
    (n >= 2), negative coordinates among them; neighbours share corners."""
    g = np.random.default_rng(seed)
    top = corners_per_axis - 2
    base = g.integers(0, top + 1, (n // 4 + 1, 3))
    near = base[g.integers(0, len(base), n)] + g.integers(-1, 2, (n, 3))
    c = np.clip(near, 0, top)
    if n > 1:
        c[0], c[-1] = 0, top
    return (c - top // 2).astype(np.int32), g.standard_normal((n, 8)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1023, 70001])
@pytest.mark.parametrize("axis", [3, 64, 1127, 1128, 1 << 20])
def test_block_edges_and_key_types(oracle, dev, n, axis):
    # 3 * 1127^3 < 2^32 < 3 * 1128^3
    coords, corners = _voxels(n, axis, 100 * n + axis)
    v, t = cubvh.sparse_marching_cubes(torch.from_numpy(coords).to(dev), torch.from_numpy(corners).to(dev), 0.1)
    assert np.array_equal(v.cpu().numpy(), oracle.sparse_mc_vertices(coords, corners, 0.1))
    assert np.array_equal(t.cpu().numpy(), oracle.sparse_mc_triangles(coords, corners, 0.1, TABLE))


@pytest.mark.gpu
@pytest.mark.parametrize("inside", [0, 255, 1, 254])
def test_uniform_blocks(oracle, dev, inside):
    """Blocks with no vertex at all, and blocks whose every voxel is cut."""
    coords = np.stack(np.meshgrid(np.arange(9), np.arange(8), np.arange(8), indexing="ij"), -1).reshape(-1, 3)
    coords = coords.astype(np.int32)
    sign = np.array([-1.0 if inside >> k & 1 else 1.0 for k in range(8)], np.float32)
    corners = np.tile(sign, (len(coords), 1))
    v, t = cubvh.sparse_marching_cubes(torch.from_numpy(coords).to(dev), torch.from_numpy(corners).to(dev), 0.0)
    if inside in (0, 255):
        assert v.shape == (0, 3) and t.shape == (0, 3)
        return
    assert np.array_equal(v.cpu().numpy(), oracle.sparse_mc_vertices(coords, corners, 0.0))
    assert np.array_equal(t.cpu().numpy(), oracle.sparse_mc_triangles(coords, corners, 0.0, TABLE))


@pytest.mark.gpu
@pytest.mark.parametrize("axis", [3, 64, 1625, 1626, 1 << 20])
def test_corner_means_of_both_key_types(oracle, dev, axis):
    # corner keys: 1625^3 < 2^32 < 1626^3
    coords, corners = _voxels(3000, axis, axis)
    off = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])
    at = (coords[:, None].astype(np.int64) + off).reshape(-1, 3)
    runs = {}
    for j, key in enumerate(map(tuple, at)):
        runs.setdefault(key, []).append(j)
    flat, mean = corners.reshape(-1), np.empty(8 * len(coords), np.float32)
    for members in runs.values():
        total = np.float32(0)
        for j in members:                        # in voxel order, in float32
            total = np.float32(total + flat[j])
        mean[members] = np.float32(total / np.float32(len(members)))
    v, t = cubvh.sparse_marching_cubes(torch.from_numpy(coords).to(dev), torch.from_numpy(corners).to(dev), 0.1,
                                       ensure_consistency=True)
    mean = mean.reshape(-1, 8)
    assert np.array_equal(v.cpu().numpy(), oracle.sparse_mc_vertices(coords, mean, 0.1))
    assert np.array_equal(t.cpu().numpy(), oracle.sparse_mc_triangles(coords, mean, 0.1, TABLE))
