"""Backward of the distance queries where its sorts begin and end, and refits
of trees of every depth.

The gradients of vertices sort the queries by face in chunks of 2^22; those of
points alone take the queries in the caller's order.  Only the queries beside
the chunks' edges get a weight, so that one left out or taken twice shows."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W
from test_grad import analytic

CHUNK = 1 << 22


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 257, CHUNK - 1, CHUNK, CHUNK + 1, 2 * CHUNK + 5])
@pytest.mark.parametrize("vertices", [False, True])
def test_backward_at_chunk_edges(oracle, dev, n, vertices):
    V, F = W.displaced_icosphere(2, 4)
    rng = np.random.default_rng(n)
    pts = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    w = np.zeros(n, np.float32)
    for at in range(0, n + 1, CHUNK):
        w[max(at - 40, 0):at + 40] = 1
    w[max(n - 40, 0):] = 1
    on = np.nonzero(w)[0]
    w[on] = rng.uniform(-1, 1, len(on)).astype(np.float32)
    bvh = cubvh.cuBVH(V, F)
    p = torch.from_numpy(pts).to(dev).requires_grad_()
    v = torch.from_numpy(V).to(dev).requires_grad_(vertices)
    d, fid, _ = bvh.unsigned_distance(p, vertices=v) if vertices else bvh.unsigned_distance(p)
    (torch.from_numpy(w).to(dev) * d).sum().backward()
    od, ofid, nn, gp, gv = analytic(oracle, V, F, pts[on], w[on].astype(np.float64))
    assert np.array_equal(fid.cpu().numpy()[on], ofid)
    got = p.grad.cpu().numpy().astype(np.float64)
    off = np.ones(n, bool)
    off[on] = False
    assert not got[off].any()
    # one double computation rounded to float, |gradient| <= 1
    assert np.abs(got[on] - gp).max() <= 2.0 ** -23
    if vertices:
        # at most len(on) terms of at most 1, each rounded once, summed in float
        lim = 2.0 ** -23 * (len(on) + 1) * np.abs(w[on]).sum() / 8
        assert np.abs(v.grad.cpu().numpy() - gv).max() <= lim and lim < 0.01


@pytest.mark.gpu
@pytest.mark.parametrize("faces", [9, 33, 257, 1280])
def test_refit_of_small_trees(oracle, dev, faces):
    V, F = W.displaced_icosphere(3, 2)
    F = F[:faces]
    bvh = cubvh.cuBVH(V, F)
    V2 = (V * np.array([1.4, 0.7, 1.0]) + np.random.default_rng(faces).normal(0, 0.02, V.shape)).astype(np.float32)
    bvh.refit(torch.from_numpy(V2).to(dev))
    pts = W.uniform_points(3000, 3)
    d, fid, _ = bvh.unsigned_distance(torch.from_numpy(pts).to(dev))
    od, ofid, _, _, _ = oracle.udf64(V2, F, pts)
    assert np.array_equal(d.cpu().numpy(), od.astype(np.float32)) and np.array_equal(fid.cpu().numpy(), ofid)
