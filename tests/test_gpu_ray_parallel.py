"""Coherent bundles of axis-parallel rays (the rays of orthographic cameras and
voxelisers) with origins exactly in planes of the boxes, against the FP64
oracle and against the same rays traced one by one between incoherent ones.
A bundle is close enough to be walked as packets: its rays have one direction
and lie within a hundredth of the mesh's extent."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh

pytestmark = pytest.mark.gpu

STEP = 2.0 ** -12     # between neighbouring rays: 32 of them stay within 0.008 of a mesh 2 wide


def _cube(k):
    """The surface of [-1, 1]^3, each side k x k squares."""
    i = np.arange(k + 1)
    corner, v, f = {}, [], []

    def at(p):
        if p not in corner:
            corner[p] = len(v)
            v.append([2.0 * c / k - 1.0 for c in p])
        return corner[p]

    for ax in range(3):
        u, w = (ax + 1) % 3, (ax + 2) % 3
        for side in (0, k):
            for a in i[:-1]:
                for b in i[:-1]:
                    q = []
                    for da, db in ((0, 0), (1, 0), (1, 1), (0, 1)):
                        p = [0, 0, 0]
                        p[ax], p[u], p[w] = side, int(a) + da, int(b) + db
                        q.append(at(tuple(p)))
                    f += [[q[0], q[1], q[2]], [q[0], q[2], q[3]]]
    return np.array(v, np.float32), np.array(f, np.int64)


def _terrain(k):
    """Steps of three heights over a regular grid of [-1, 1]^2, with the walls between them."""
    h = lambda a, b: 0.25 * ((a // 2 + b // 3) % 3)
    v, f = [], []

    def quad(*ps):
        n = len(v)
        v.extend(ps)
        f.extend([[n, n + 1, n + 2], [n, n + 2, n + 3]])

    c = [2.0 * a / k - 1.0 for a in range(k + 1)]
    for a in range(k):
        for b in range(k):
            z = h(a, b)
            quad((c[a], c[b], z), (c[a + 1], c[b], z), (c[a + 1], c[b + 1], z), (c[a], c[b + 1], z))
            if a + 1 < k and h(a + 1, b) != z:
                quad((c[a + 1], c[b], z), (c[a + 1], c[b + 1], z), (c[a + 1], c[b + 1], h(a + 1, b)),
                     (c[a + 1], c[b], h(a + 1, b)))
            if b + 1 < k and h(a, b + 1) != z:
                quad((c[a], c[b + 1], z), (c[a + 1], c[b + 1], z), (c[a + 1], c[b + 1], h(a, b + 1)),
                     (c[a], c[b + 1], h(a, b + 1)))
    return np.array(v, np.float32), np.array(f, np.int64)


MESHES = {"box": lambda: _cube(1), "cube": lambda: _cube(8), "terrain": lambda: _terrain(16)}


def _bundles(planes, axis, sign, shape):
    """Bundles of 32 rays along an axis: a row at each plane of a crossing axis, a 4 x 8 grid that starts or ends
    at a pair of planes, and 32 times one ray through a vertex."""
    u, w = [k for k in range(3) if k != axis]
    out = []
    j = np.arange(32)
    for a in planes[u]:
        for b in planes[w]:
            sa = -1.0 if a == planes[u][-1] else 1.0       # rows run along the mesh, not past its end
            sb = -1.0 if b == planes[w][-1] else 1.0
            o = np.zeros((32, 3))
            o[:, axis] = -3.0 * sign
            if shape == "row":
                o[:, u] = a
                o[:, w] = b + sb * (0.1 + j * STEP)
            elif shape == "grid":
                o[:, u] = a + sa * (j // 8) * STEP
                o[:, w] = b + sb * (j % 8) * STEP
            else:
                o[:, u], o[:, w] = a, b
            out.append(o)
    return np.array(out, np.float32)


def _packets(v, o, d):
    """Every 32 rays of o are one coherent packet: units of 8 rays within 0.8 % of the mesh's extent, one direction."""
    assert (np.ptp(o, axis=1) <= 0.008 * np.ptp(v, axis=0).max()).all()
    assert np.ptp(d, axis=0).max() <= 1e-6


def _planes(v):
    return [np.unique(v[:, k])[[0, len(np.unique(v[:, k])) // 2, -1]] for k in range(3)]


def _trace(bvh, o, d, dev):
    return [t.cpu().numpy() for t in bvh.ray_trace(torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev))]


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("shape", ["row", "grid", "point"])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_axis_parallel_bundles(oracle, dev, mesh, shape, axis, sign):
    v, f = MESHES[mesh]()
    bvh = cubvh.cuBVH(v, f)
    bundles = _bundles(_planes(v), axis, sign, shape)
    d1 = np.zeros((32, 3), np.float32)
    d1[:, axis] = sign
    _packets(v, bundles, d1)
    o, d = bundles.reshape(-1, 3), np.tile(d1, (len(bundles), 1))
    ot, ofid, _ = oracle.ray64(v, f, o, d)
    assert (ofid >= 0).any()
    pos = (o.astype(np.float64) + ot[:, None] * d.astype(np.float64)).astype(np.float32)
    want = [pos, ofid, ot.astype(np.float32)]
    for k in range(len(bundles)):                    # a call a bundle: one packet
        got = _trace(bvh, bundles[k], d1, dev)
        for x, y in zip(got, want):
            assert np.array_equal(x, y[32 * k:32 * k + 32]), (k, bundles[k][0])
    # each ray in a unit with seven of other directions: rays on their own
    rng = np.random.default_rng(3)
    n = len(o)
    o8 = rng.uniform(-2, 2, (n, 8, 3)).astype(np.float32)
    d8 = rng.standard_normal((n, 8, 3)).astype(np.float32)
    o8[:, 3], d8[:, 3] = o, d
    got = _trace(bvh, o8.reshape(-1, 3), d8.reshape(-1, 3), dev)
    for x, y in zip(got, want):
        assert np.array_equal(x.reshape((n, 8) + x.shape[1:])[:, 3], y)


@pytest.mark.parametrize("tiny", [0.0, 1e-14, 1e-20, 1e-31, 1e-40])
@pytest.mark.parametrize("out", [1.0, -1.0])
def test_all_but_parallel(oracle, dev, tiny, out):
    """A component that the double test does not see against the origin: outwards or inwards of the plane, in all
    rays of a bundle and in some."""
    v, f = _cube(4)
    bvh = cubvh.cuBVH(v, f)
    j = np.arange(32)
    for axis in range(3):
        u, w = [k for k in range(3) if k != axis]
        for side in (-1.0, 1.0):
            for some in (32, 5):
                o = np.zeros((32, 3), np.float32)
                d = np.zeros((32, 3), np.float32)
                o[:, axis], o[:, u], o[:, w] = 3.0, side, 0.1 + j * STEP
                d[:, axis] = -1.0
                d[j % some == 0 if some < 32 else slice(None), u] = out * side * tiny
                _packets(v, o[None], d)
                ot, ofid, _ = oracle.ray64(v, f, o, d)
                _, fid, depth = _trace(bvh, o, d, dev)
                assert np.array_equal(depth, ot.astype(np.float32)) and np.array_equal(fid, ofid)


def test_orthographic_grid(oracle, dev):
    """A whole orthographic image whose border and every 32nd line lie in planes of the mesh, and the same rays in
    another order and in parts."""
    v, f = _cube(8)
    bvh = cubvh.cuBVH(v, f)
    x = np.linspace(-1.0, 1.0, 257)                  # pixels 1/128 apart: units 0.055 wide are rays on their own,
    fine = np.concatenate([np.arange(64) * STEP - 1.0, 1.0 - np.arange(64)[::-1] * STEP])   # fine ones packets
    for axis in range(3):
        for g in (x, fine):
            a, b = np.meshgrid(g, g, indexing="ij")
            o = np.full((a.size, 3), 2.0, np.float32)
            u, w = [k for k in range(3) if k != axis]
            o[:, u], o[:, w] = a.ravel(), b.ravel()
            d = np.zeros_like(o)
            d[:, axis] = -1.0
            ot, ofid, _ = oracle.ray64(v, f, o, d)
            assert (ofid >= 0).all()
            got = _trace(bvh, o, d, dev)
            assert np.array_equal(got[1], ofid) and np.array_equal(got[2], ot.astype(np.float32))
            p = np.random.default_rng(axis).permutation(len(o))
            mixed = _trace(bvh, np.ascontiguousarray(o[p]), np.ascontiguousarray(d[p]), dev)
            for s, t in zip(got, mixed):
                assert np.array_equal(s[p], t)
            parts = [_trace(bvh, o[i:i + 1000], d[i:i + 1000], dev) for i in range(0, len(o), 1000)]
            for k in range(3):
                assert np.array_equal(got[k], np.concatenate([q[k] for q in parts]))
