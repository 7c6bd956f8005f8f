"""Point queries whose packets walk long (points about equally far from very many
triangles) in calls of few to very many such packets: the results of small
calls, bit for bit, and what such a call costs."""

import numpy as np
import pytest
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_536, 70_001, 200_000])
@pytest.mark.parametrize("spread", [0.0, 0.01, 0.3])
@pytest.mark.parametrize("share", [0.1, 1.0])
def test_long_walks(dev, n, spread, share):
    """share of the points around the middle, the others in the box, against calls of 50,000 points (no packets)."""
    rng = np.random.default_rng(n)
    pts = W.uniform_points(n, 3)
    mid = rng.random(n) < share
    pts[mid] = (rng.uniform(-1, 1, (int(mid.sum()), 3)) * spread).astype(np.float32)
    p = torch.from_numpy(pts).to(dev)
    bvh = cubvh.cuBVH(*W.displaced_icosphere(5, 3))
    d, f, u = bvh.unsigned_distance(p, return_uvw=True)
    parts = [bvh.unsigned_distance(q.contiguous(), return_uvw=True) for q in p.split(50_000)]
    for got, want in zip((d, f, u), zip(*parts)):
        assert torch.equal(got, torch.cat(want))


def test_long_walks_cost(dev):
    """100,003 points in one place: 1.7 times uniform ones; 5 times with a warp for each of them."""
    bvh = cubvh.cuBVH(*W.displaced_icosphere(5, 3))
    box = torch.from_numpy(W.uniform_points(100_003, 2)).to(dev)

    def ms(p):
        t = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            bvh.unsigned_distance(p)
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return min(t)

    assert ms(torch.zeros_like(box)) < 3 * ms(box)
