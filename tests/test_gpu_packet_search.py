"""The packet distance search at the edges of its shapes, against the FP64
oracle bit for bit: partial packets, points that take no part in the walk,
candidate lists that overflow (more triangles at one distance than fit)."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(oracle, v, f, pts, dev):
    d, fid, uvw = cubvh.cuBVH(v, f).unsigned_distance(torch.from_numpy(pts).to(dev), return_uvw=True)
    od, ofid, ouvw, _, _ = oracle.udf64(v, f, pts)
    assert np.array_equal(d.cpu().numpy(), od.astype(np.float32))
    assert np.array_equal(fid.cpu().numpy(), ofid)
    assert np.array_equal(uvw.cpu().numpy(), ouvw.astype(np.float32))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 2367, 2368, 2369, 4737, 65535, 65536, 65567])
def test_packet_edges(oracle, dev, n):
    """Below 65,536 points eight lanes a query, one, two or four queries a warp; above, packets of 32."""
    v, f = W.displaced_icosphere(2, 2)
    _check(oracle, v, f, W.uniform_points(n, n), dev)


def _fan(valence, copies):
    """A cone of `valence` triangles around one apex, every face `copies` times, and a far tetrahedron-like strip."""
    a = np.arange(valence) * (2 * np.pi / valence)
    v = np.concatenate([[[0, 0, 0.5]], np.stack([np.cos(a), np.sin(a), 0 * a], 1)]).astype(np.float32)
    f = np.stack([np.zeros(valence, int), 1 + np.arange(valence), 1 + (np.arange(valence) + 1) % valence], 1)
    return v, np.tile(f, (copies, 1)).astype(np.int64)


@pytest.mark.parametrize("valence,copies", [(40, 1), (8, 12), (200, 2)])
@pytest.mark.parametrize("n", [40, 5000, 70000])
def test_candidate_overflow(oracle, dev, valence, copies, n):
    """Points above the apex tie on every triangle of the fan."""
    v, f = _fan(valence, copies)
    rng = np.random.default_rng(valence + n)
    top = np.array([0, 0, 1.0]) + rng.uniform(-0.05, 0.05, (n // 2, 3))
    pts = np.concatenate([top, rng.uniform(-1, 1, (n - n // 2, 3))]).astype(np.float32)
    _check(oracle, v, f, pts, dev)


@pytest.mark.parametrize("counts", [[1, 0, 300, 7], [40000, 0, 25536, 3]])
def test_small_and_large_arenas(oracle, dev, counts):
    """Queries of several meshes, one of them without any, on both sides of the split."""
    meshes = [W.icosphere(2, 0.8), W.displaced_icosphere(2, 1), W.displaced_icosphere(3, 3), W.icosphere(1, 0.5)]
    arena = cubvh.BVHArena(meshes)
    arena.set_queries(counts, ["unsigned", "watertight", "watertight", "raystab"])
    qs = [W.uniform_points(n, i) for i, n in enumerate(counts)]
    d, fid, uvw = arena.distance(torch.from_numpy(np.concatenate(qs)).to(dev), return_uvw=True)
    at = 0
    for (v, f), q, mode in zip(meshes, qs, ["unsigned", "watertight", "watertight", "raystab"]):
        if len(q):
            bvh, p = cubvh.cuBVH(v, f), torch.from_numpy(q).to(dev)
            want = (bvh.unsigned_distance(p, return_uvw=True) if mode == "unsigned"
                    else bvh.signed_distance(p, return_uvw=True, mode=mode))
            for a, b in zip((d, fid, uvw), want):
                assert torch.equal(a[at:at + len(q)], b)
            od, ofid, _, _, _ = oracle.udf64(v, f, q[:2000])
            assert np.array_equal(fid[at:at + len(q)][:2000].cpu().numpy(), ofid)
            assert np.array_equal(d[at:at + len(q)][:2000].abs().cpu().numpy(), od.astype(np.float32))
        at += len(q)


def test_idle_points(oracle, dev):
    """Points that are no number, infinite or out of reach, between ordinary ones in the same packets."""
    v, f = W.displaced_icosphere(3, 2)
    pts = W.uniform_points(70016, 5)
    odd = np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, -np.inf, 0], [3e38, 0, 0], [2000, 0, 0], [0, 1.5e3, 0]], np.float32)
    at = np.arange(0, len(pts), 37)
    mixed = pts.copy()
    mixed[at] = odd[np.arange(len(at)) % len(odd)]
    bvh = cubvh.cuBVH(v, f)
    for n in (len(pts), 4096, 300):
        want = bvh.unsigned_distance(torch.from_numpy(pts[:n]).to(dev))
        d, fid, _ = bvh.unsigned_distance(torch.from_numpy(mixed[:n]).to(dev))
        keep = np.ones(n, bool)
        keep[at[at < n]] = False
        keep = torch.from_numpy(keep).to(dev)
        assert torch.equal(d[keep], want[0][keep]) and torch.equal(fid[keep], want[1][keep])
        assert bool((d[~keep] == 0).all()) and bool((fid[~keep] == 0).all())
