"""Ray packets at the edges of their shapes, against the FP64 oracle bit for
bit: partial packets, units whose directions change sign or have zero
components, rays that are not finite inside a coherent unit, hit lists that
overflow, and bundles from parallel to incoherent (the split between packets
and lanes)."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(oracle, v, f, o, d, dev):
    pos, fid, depth = cubvh.cuBVH(v, f).ray_trace(torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev))
    ot, ofid, _ = oracle.ray64(v, f, o, d)
    assert np.array_equal(depth.cpu().numpy(), ot.astype(np.float32))
    assert np.array_equal(fid.cpu().numpy(), ofid)
    want = (o.astype(np.float64) + ot[:, None] * d.astype(np.float64)).astype(np.float32)
    assert np.array_equal(pos.cpu().numpy(), want)
    return ofid


def _bundle(n, spread, seed, axis=None):
    """Rays from (0.1, 0.05, 2.5) about the origin's direction, or about an axis plane."""
    rng = np.random.default_rng(seed)
    o = np.tile(np.array([[0.1, 0.05, 2.5]]), (n, 1))
    d = -o + rng.uniform(-0.5, 0.5, (1, 3)) + rng.standard_normal((n, 3)) * spread
    if axis is not None:
        d[:, axis] = rng.standard_normal(n) * 1e-4   # signs change within a unit
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 31, 32, 33, 100, 8193])
def test_partial_packets(oracle, dev, n):
    v, f = W.displaced_icosphere(3, 2)
    o, d = _bundle(n, 1e-3, n)
    _check(oracle, v, f, o, d, dev)


@pytest.mark.parametrize("spread", [0.0, 1e-4, 2e-3, 4e-3, 8e-3, 0.02, 0.2])
@pytest.mark.parametrize("axis", [None, 0, 1])
def test_bundles(oracle, dev, spread, axis):
    v, f = W.displaced_icosphere(3, 2)
    o, d = _bundle(2000, spread, 7, axis)
    assert (_check(oracle, v, f, o, d, dev) >= 0).any()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1, -1])
def test_parallel_rays(oracle, dev, axis, sign):
    """Zero direction components, origins on a grid that meets vertices and box planes."""
    v, f = W.icosphere(2, 0.75)
    x = np.linspace(-0.75, 0.75, 33)
    g = np.stack(np.meshgrid(x, x, indexing="ij"), -1).reshape(-1, 2)
    o, d = np.zeros((len(g), 3)), np.zeros((len(g), 3))
    o[:, [k for k in range(3) if k != axis]] = g
    o[:, axis] = -2.0 * sign
    d[:, axis] = sign
    _check(oracle, v, f, o.astype(np.float32), d.astype(np.float32), dev)


def test_odd_rays_inside_units(oracle, dev):
    """Rays 1, 2, 4, 5, 6 of a unit are not looked at when units are judged."""
    v, f = W.displaced_icosphere(3, 2)
    o, d = _bundle(1024, 1e-3, 3)
    want = cubvh.cuBVH(v, f).ray_trace(torch.from_numpy(o).to(dev), torch.from_numpy(d).to(dev))
    o2, d2 = o.copy(), d.copy()
    odd = np.arange(1, 1024, 8)
    for k, (arr, val) in enumerate([(o2, np.nan), (d2, np.nan), (d2, 0.0), (o2, np.inf), (d2, [-1, 0, 0])]):
        arr[odd[k::7] + (k % 2)] = val
    changed = np.zeros(1024, bool)
    for k in range(5):
        changed[odd[k::7] + (k % 2)] = True
    got = cubvh.cuBVH(v, f).ray_trace(torch.from_numpy(o2).to(dev), torch.from_numpy(d2).to(dev))
    keep = torch.from_numpy(~changed).to(dev)
    for a, b in zip(got, want):
        assert torch.equal(a[keep], b[keep])
    aside = odd[4::7]          # the unit's stray ray is traced as any other
    ot, ofid, _ = oracle.ray64(v, f, o2[aside], d2[aside])
    assert np.array_equal(got[1].cpu().numpy()[aside], ofid)


@pytest.mark.parametrize("copies", [9, 30])
def test_hit_list_overflow(oracle, dev, copies):
    """Every face many times: more equal hits than a list holds, the lowest face index wins."""
    v, f = W.icosphere(1, 0.75)
    o, d = _bundle(500, 1e-3, 5)
    _check(oracle, v, np.tile(f, (copies, 1)), o, d, dev)
