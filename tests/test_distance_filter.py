"""The FP32 distance filter of the packet search (tri_d2_w, geom.cuh) in
numpy float32, with a triangle's frame as k_expand_tris makes it, against
exact squared distances in extended precision: the error stays within
8e-6 (|p - a|^2 + L^2) for slivers and segments too."""

import numpy as np
import pytest

f32 = np.float32


def _frame(A, B, C):
    A, B, C = (x.astype(np.float64) for x in (A, B, C))
    l = np.stack([((B - A) ** 2).sum(1), ((C - B) ** 2).sum(1), ((A - C) ** 2).sum(1)], 1)
    k = np.where((l[:, 1] > l[:, 0]) & (l[:, 1] >= l[:, 2]), 1, np.where(l[:, 2] > l[:, 0], 2, 0))
    P, i = np.stack([A, B, C], 1), np.arange(len(A))
    A, B, C = P[i, k], P[i, (k + 1) % 3], P[i, (k + 2) % 3]
    e = B - A
    L = np.linalg.norm(e, axis=1)
    ex = e / L[:, None]
    w = C - A
    cx = (w * ex).sum(1)
    r = w - ex * cx[:, None]
    cy = np.linalg.norm(r, axis=1)
    good = cy > 1e-9 * L
    ey = r / np.where(good, cy, 1)[:, None]
    ey -= ex * (ey * ex).sum(1)[:, None]
    ey = np.where(good[:, None], ey, np.cross(np.eye(3)[np.abs(ex).argmin(1)], ex))
    cy = np.where(good, cy, 0)
    ey /= np.linalg.norm(ey, axis=1, keepdims=True)
    ac, bx = np.hypot(cx, cy), cx - L
    bc = np.hypot(bx, cy)
    one = np.array([1.0, 0.0])
    v = np.where(ac[:, None] > 0, np.stack([cx, cy], 1) / np.where(ac, ac, 1)[:, None], one)
    u = np.where(bc[:, None] > 0, np.stack([bx, cy], 1) / np.where(bc, bc, 1)[:, None], one)
    return [x.astype(f32) for x in (A, L, ex, ac, ey, bc, v, u)]


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f32)


def _filter(p, t):
    a, L, ex, lac, ey, lbc, v, u = t
    qx, qy, qz = (p - a).T
    x = _fma(qz, ex[:, 2], _fma(qy, ex[:, 1], qx * ex[:, 0]))
    y = _fma(qz, ey[:, 2], _fma(qy, ey[:, 1], qx * ey[:, 0]))
    qq = _fma(qz, qz, _fma(qy, qy, qx * qx))
    xb = x - L

    def over(s, l):
        return np.maximum(np.maximum(-s, l), f32(0))

    s1, c1 = _fma(y, v[:, 1], x * v[:, 0]), _fma(x, v[:, 1], -(y * v[:, 0]))
    s2, c2 = _fma(y, u[:, 1], xb * u[:, 0]), _fma(y, u[:, 0], -(xb * u[:, 1]))
    o0, o1, o2 = over(x, xb), over(s1, s1 - lac), over(s2, s2 - lbc)
    m = np.minimum(np.minimum(_fma(o0, o0, y * y), _fma(o1, o1, c1 * c1)), _fma(o2, o2, c2 * c2))
    inside = np.minimum(np.minimum(np.minimum(y, c1), np.minimum(c2, x)), -xb) >= 0
    h2 = np.maximum(_fma(-y, y, _fma(-x, x, qq)), f32(0))
    return h2 + np.where(inside, f32(0), m), f32(8e-6) * _fma(L, L, qq)


def _exact(p, A, B, C):
    p, A, B, C = (x.astype(np.longdouble) for x in (p, A, B, C))

    def seg(a, b):
        e = b - a
        ee = (e * e).sum(1)
        t = np.clip(np.where(ee > 0, ((p - a) * e).sum(1) / np.where(ee > 0, ee, 1), 0), 0, 1)
        return ((p - a - e * t[:, None]) ** 2).sum(1)

    d = np.minimum(np.minimum(seg(A, B), seg(B, C)), seg(C, A))
    n = np.cross(B - A, C - A)
    nn = (n * n).sum(1)
    inside = nn > 0
    for a, b in ((A, B), (B, C), (C, A)):
        inside &= (np.cross(b - a, p - a) * n).sum(1) >= 0
    h = ((p - A) * n).sum(1)
    return np.where(inside, np.minimum(d, h * h / np.where(nn > 0, nn, 1)), d)


@pytest.mark.parametrize("kind", ["ordinary", "sliver", "needle", "segment", "far"])
@pytest.mark.parametrize("near", [False, True])
def test_filter_bound(kind, near):
    rng = np.random.default_rng([len(kind), near])
    n = 40000
    scale = 10 ** rng.uniform(-3, 1, (n, 1))
    off = rng.uniform(-1, 1, (n, 3)) * (10 ** rng.uniform(-2, 3, (n, 1)) if kind == "far" else 1)
    A, B = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    C = rng.standard_normal((n, 3))
    if kind in ("sliver", "needle", "segment"):
        t = rng.uniform(-0.2, 1.2, (n, 1))
        t = np.round(t) if kind == "needle" else t
        C = A + (B - A) * t + (0 if kind == "segment" else rng.standard_normal((n, 3)) * 10 ** rng.uniform(-8, 0, (n, 1)))
    A, B, C = ((x * scale + off).astype(f32) for x in (A, B, C))
    if near:
        w = rng.dirichlet([0.5, 0.5, 0.5], n)
        base = A * w[:, :1] + B * w[:, 1:2] + C * w[:, 2:]
    else:   # around an edge's line, past its ends
        base = A + (B - A) * rng.uniform(-1, 2, (n, 1))
    p = (base + rng.standard_normal((n, 3)) * scale * 10 ** rng.uniform(-8, 1, (n, 1))).astype(f32)
    d2, err = _filter(p, _frame(A, B, C))
    off_by = np.abs(d2 - _exact(p, A, B, C))
    assert (off_by <= err).all(), float((off_by / err).max())
