"""Watertight signs where the normal sum's members are certain by the FP32 test
and where they are not: closest points on vertices, edges and faces, some at
the sum's radius (1e-3) from a vertex or an edge, queries from on the surface
to far away; smooth and sharp meshes, right angles, faces of either
orientation side by side, two sheets within the radius, faces of no area.
Signs equal the FP64 oracle's wherever it calls them decided."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cube(n):
    """A cube of side 1 around the origin, n x n quads a side."""
    g = np.linspace(-0.5, 0.5, n + 1)
    V, F = [], []
    for axis in range(3):
        for side in (-0.5, 0.5):
            at = len(V)
            for a in g:
                for b in g:
                    p = [0.0, 0.0, 0.0]
                    p[axis], p[(axis + 1) % 3], p[(axis + 2) % 3] = side, a, b
                    V.append(p)
            for i in range(n):
                for j in range(n):
                    q = [at + i * (n + 1) + j, at + (i + 1) * (n + 1) + j, at + (i + 1) * (n + 1) + j + 1,
                         at + i * (n + 1) + j + 1]
                    if side < 0:
                        q = q[::-1]
                    F += [[q[0], q[1], q[2]], [q[0], q[2], q[3]]]
    return np.array(V, np.float32), np.array(F, np.int32)


def _mesh(name):
    V, F = W.displaced_icosphere(3, 6)
    rng = np.random.default_rng(3)
    if name == "cube":
        return _cube(5)
    if name == "flat":
        return (V * np.array([1, 0.2, 0.05])).astype(np.float32), F
    if name == "sheets":
        return (V * np.array([1, 1, 0.0012])).astype(np.float32), F
    if name == "needles":
        return (V * np.array([1, 0.004, 0.3])).astype(np.float32), F
    if name == "flipped":
        F = F.copy()
        k = rng.choice(len(F), len(F) // 5, replace=False)
        F[k] = F[k][:, ::-1]
    if name == "collapsed":
        V = V.copy()
        for t in rng.choice(len(F), 30, replace=False):
            V[F[t, 1]] = V[F[t, 0]]
    return V, F


@pytest.mark.parametrize("name", ["smooth", "cube", "flat", "sheets", "needles", "flipped", "collapsed"])
def test_signs(oracle, dev, name):
    V, F = _mesh(name)
    rng = np.random.default_rng(11)
    tri = V[F].astype(np.float64)
    lam = rng.dirichlet([1, 1, 1], len(F))
    mid, cen = 0.5 * (tri[:, 0] + tri[:, 1]), tri.mean(1)
    on = [V.astype(np.float64), mid, np.einsum("nk,nkj->nj", lam, tri)]
    for corner in (tri[:, 0], mid):              # 1e-3 from a corner or an edge, a little less, a little more
        u = cen - corner
        u /= np.maximum(np.linalg.norm(u, axis=1, keepdims=True), 1e-12)
        on.append(corner + 1e-3 * rng.uniform(0.998, 1.002, (len(u), 1)) * u)
    on = np.concatenate(on)
    pts = [W.uniform_points(2000, 8).astype(np.float64)]
    for h in (0.0, 1e-7, 1e-5, 3e-4, 1e-3, 1e-2, 0.3):
        u = rng.normal(size=on.shape)
        pts.append((on + h * u / np.linalg.norm(u, axis=1, keepdims=True))[rng.random(len(on)) < 0.5])
    pts = np.concatenate(pts).astype(np.float32)
    bvh = cubvh.cuBVH(V, F)
    d, fid, _ = bvh.signed_distance(torch.from_numpy(pts).to(dev), mode="watertight")
    d, fid = d.cpu().numpy(), fid.cpu().numpy()
    want, ofid, flags = oracle.sdf_watertight64(V, F, pts)
    want = want.astype(np.float32)
    assert np.array_equal(fid, ofid) and np.array_equal(np.abs(d), np.abs(want))
    ok = (flags & 1) == 0     # the sum's dot product is not zero to 1e-12
    assert ok.mean() > 0.5
    assert np.array_equal(np.signbit(d[ok]), np.signbit(want[ok]))
