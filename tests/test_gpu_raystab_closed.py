"""Raystab signs of closed and open meshes, against the FP64 oracle (all 64
rays): closed meshes end inside points after one ray by the parity of its
crossings, open ones trace every ray; nested and overlapping closed shells
(even parities inside), points on the surface, far away and after a refit
that keeps or breaks the closedness."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _merge(*meshes):
    vs, fs, at = [], [], 0
    for v, f in meshes:
        vs.append(np.asarray(v, np.float32))
        fs.append(np.asarray(f, np.int64) + at)
        at += len(v)
    return np.concatenate(vs), np.concatenate(fs)


def _mesh(name):
    v, f = W.displaced_icosphere(3, 4)
    if name == "closed":
        return v, f
    if name == "one_face_missing":
        return v, f[:-1]
    if name == "one_face_twice":
        return v, np.concatenate([f, f[:1]])
    if name == "all_faces_twice":
        return v, np.concatenate([f, f])
    if name == "nested":
        return _merge(W.icosphere(3, 0.9), W.icosphere(3, 0.5))
    if name == "overlapping":
        a, b = W.icosphere(3, 0.6), W.icosphere(2, 0.6)
        return _merge((a[0] - np.float32(0.3), a[1]), (b[0] + np.float32(0.3), b[1]))
    if name == "unshared_vertices":   # closed by position only
        return v[f].reshape(-1, 3), np.arange(3 * len(f)).reshape(-1, 3)
    if name == "far":                  # crossings past t = 1000
        return (v * np.float32(1500)).astype(np.float32), f
    raise KeyError(name)


def _points(v, f, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = v.min(0), v.max(0)
    box = rng.uniform(lo - 0.1 * (hi - lo), hi + 0.1 * (hi - lo), (n, 3))
    on = np.concatenate([v[f[:40]].mean(1), v[:40], (v[f[:40, 0]] + v[f[:40, 1]]) / 2])   # faces, vertices, edges
    return np.concatenate([box, on]).astype(np.float32)


@pytest.mark.parametrize("name", ["closed", "one_face_missing", "one_face_twice", "all_faces_twice", "nested",
                                  "overlapping", "unshared_vertices", "far"])
def test_signs_equal_oracle(oracle, dev, stab_dirs, name):
    v, f = _mesh(name)
    pts = _points(v, f, 3000, 8)
    d, fid, _ = cubvh.cuBVH(v, f).signed_distance(torch.from_numpy(pts).to(dev), mode="raystab")
    sd, ofid, _ = oracle.sdf_raystab64(v, f, pts, dirs=stab_dirs(len(pts)))
    assert np.array_equal(d.cpu().numpy(), sd.astype(np.float32))
    assert np.array_equal(fid.cpu().numpy(), ofid)


@pytest.mark.parametrize("device_build", [False, True])
def test_arena_mixes_closed_and_open(oracle, dev, stab_dirs, device_build):
    names = ["closed", "one_face_missing", "nested", "closed"]
    meshes = [_mesh(n) for n in names]
    qs = [_points(v, f, 700 + 31 * i, i) for i, (v, f) in enumerate(meshes)]
    arena = cubvh.BVHArena(meshes, device_build=device_build)
    arena.set_queries([len(q) for q in qs], ["raystab"] * len(qs))
    pts = torch.from_numpy(np.concatenate(qs)).to(dev)
    for _ in range(2):   # the parities start from zero in every call
        d = arena.distance(pts)[0].cpu().numpy()
        at = 0
        for (v, f), q in zip(meshes, qs):
            sd, _, _ = oracle.sdf_raystab64(v, f, q, dirs=stab_dirs(len(q)))
            assert np.array_equal(d[at:at + len(q)], sd.astype(np.float32))
            at += len(q)


def test_refit_that_tears_the_mesh(oracle, dev, stab_dirs):
    """Vertices of a soup moved apart: closed before, open after."""
    v, f = _mesh("unshared_vertices")
    bvh = cubvh.cuBVH(v, f)
    pts = _points(v, f, 2000, 9)
    torn = v.copy()
    torn[:300] *= np.float32(1.5)
    for verts in (v, torn, v):
        d = bvh.signed_distance(torch.from_numpy(pts).to(dev), mode="raystab",
                                vertices=torch.from_numpy(verts).to(dev))[0]
        sd, _, _ = oracle.sdf_raystab64(verts, f, pts, dirs=stab_dirs(len(pts)))
        assert np.array_equal(d.cpu().numpy(), sd.astype(np.float32))
