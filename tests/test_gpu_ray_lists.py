"""Rays with more possible closest hits than their list of candidates holds,
each walked alone (a unit of eight with seven rays of other directions) and in
packets, against the FP64 oracle."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh

pytestmark = pytest.mark.gpu


def _cube(copies):
    v = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    quads = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    f = np.array([t for a, b, c, d in quads for t in ((a, b, c), (a, c, d))], np.int64)
    return v, np.tile(f, (copies, 1))


def _check(oracle, v, f, o, d, got):
    ot, ofid, _ = oracle.ray64(v, f, o, d)
    assert (ofid >= 0).any()
    assert np.array_equal(got[2].cpu().numpy(), ot.astype(np.float32))
    assert np.array_equal(got[1].cpu().numpy(), ofid)


@pytest.mark.parametrize("copies", [1, 2, 4, 5, 9, 20])
@pytest.mark.parametrize("tiny", [1e-14, 1e-20, 1e-31])
@pytest.mark.parametrize("third", [0.03125, 0.0])
def test_rays_alone_in_a_plane(oracle, dev, copies, tiny, third):
    """Along the sides of a cube, with a component away from them or towards them that the double test hardly sees."""
    v, f = _cube(copies)
    rng = np.random.default_rng(copies)
    o, d = [], []
    for axis in range(3):
        u, w = [k for k in range(3) if k != axis]
        for side in (-1.0, 1.0):
            for out in (-1.0, 1.0):
                for x in (-0.9, -0.3, 0.2, 0.7):
                    p, q = np.zeros(3), np.zeros(3)
                    p[axis], p[u], p[w] = 3.0, side, x
                    q[axis], q[u], q[w] = -1.0, out * tiny, third
                    o.append(p)
                    d.append(q)
    o, d = np.array(o, np.float32), np.array(d, np.float32)
    n = len(o)
    o8 = rng.uniform(-2, 2, (n, 8, 3)).astype(np.float32)
    d8 = rng.standard_normal((n, 8, 3)).astype(np.float32)
    o8[:, 3], d8[:, 3] = o, d
    got = cubvh.cuBVH(v, f).ray_trace(torch.from_numpy(o8.reshape(-1, 3)).to(dev), torch.from_numpy(d8.reshape(-1, 3)).to(dev))
    _check(oracle, v, f, o, d, [g.view(n, 8, -1)[:, 3].squeeze(-1) for g in got])


@pytest.mark.parametrize("copies", [1, 2, 4, 5, 9, 20])
def test_packets_with_full_lists(oracle, dev, copies):
    """Bundles over an edge and a corner of the cube: some lists of a packet fill, several times, others do not."""
    v, f = _cube(copies)
    j = np.arange(64)
    o, d = np.zeros((64, 3)), np.zeros((64, 3))
    o[:] = (2.5, 2.0, 3.0)
    d[:] = np.array([1.0, 1.0, 1.0]) - o[0] + np.stack([(j // 8 - 3) * 1e-3, (j % 8 - 4) * 1e-3, 0 * j], 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o, d = o.astype(np.float32), d.astype(np.float32)
    got = cubvh.cuBVH(v, f).ray_trace(torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev))
    _check(oracle, v, f, o, d, got)
