"""Workloads of the public query path for timing and comparison.

``listed()`` names the workloads, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (device tensors, the
BVH handle), ``run`` is one pass through the public entry points, ``work`` the
bytes and operations that pass cannot do without, and ``exact`` the same
outputs in 64 bits by brute force (plain torch) where that is affordable.

Meshes come from ``cubvh_b200.workloads`` (icospheres, displaced icospheres,
tori); query sets are drawn on the GPU with the distributions that module
describes (uniform, uniform + near-surface band, dilated box, pinhole cameras,
incoherent rays, dense grids).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import cubvh_b200 as cubvh
from cubvh_b200 import workloads as W

DEV = "cuda"
MAX_PAIRS = 2.0e10   # query x face pairs that exact() may visit


def listed():
    return [
        # one small batch, as an interactive tool or a per-frame probe sends it: launches and latency
        dict(name="udf_uvw_1k", op="distance", mode="unsigned", mesh="icosphere", level=4, points=1000,
             where="uniform", uvw=True),
        # sampling a field around a small mesh with the closest point (uvw), one million points
        dict(name="udf_uvw_1m", op="distance", mode="unsigned", mesh="icosphere", level=4, points=1 << 20,
             where="uniform", uvw=True),
        # the voxelisation recipe: the distance field of open tori on a dense grid
        dict(name="udf_grid_384", op="distance", mode="unsigned", mesh="tori", level=0, points=384 ** 3,
             where="grid", uvw=False),
        # training points of a neural SDF: half uniform, half near the surface, watertight sign
        dict(name="sdf_watertight_8m", op="distance", mode="watertight", mesh="displaced", level=6,
             points=8 << 20, where="mixed", uvw=False),
        # sign by stab rays (meshes that are not watertight), points of the dilated bounding box
        dict(name="sdf_raystab_2m", op="distance", mode="raystab", mesh="displaced", level=6, points=2 << 20,
             where="box", uvw=False),
        # rendering: pinhole cameras, rays stored row by row
        dict(name="rays_camera_33m", op="rays", kind="camera", level=6, poses=8, width=2048, height=2048),
        # visibility and path tracing bounces: rays without any coherence, an odd count
        dict(name="rays_random_5m", op="rays", kind="random", level=6, poses=1, width=5000001, height=1),
        # fitting a mesh: refit to moved vertices, distance, gradients of points and vertices
        dict(name="gradient_4m", op="gradient", mode="unsigned", level=6, points=4 << 20),
        # a dataset of many meshes in one batch, forward and backward (points), half of them signed
        dict(name="arena_48", op="arena", meshes=48, max_level=6, min_points=10000, max_points=200000),
        # free-space components of a 512^3 occupancy grid
        dict(name="floodfill_512", op="floodfill", b=1, h=512, w=512, d=512),
        # occupancy to signed distance on small ragged volumes, rows that are no multiple of 32
        dict(name="udf_to_sdf_ragged", op="udf_to_sdf", b=2, h=181, w=203, d=197),
        # surface extraction from a sparse band of voxels
        dict(name="marching_cubes_192", op="marching_cubes", res=192, average=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["unsigned", "unsigned", "grid", "watertight", "watertight", "raystab", "camera", "camera",
                     "random", "gradient", "arena", "floodfill", "udf_to_sdf", "marching_cubes"])
    if op == "unsigned":
        return dict(op="distance", mode="unsigned", mesh=rng.choice(["icosphere", "displaced", "tori"]),
                    level=rng.randint(2, 6), points=_log(rng, 1000, 8 << 20),
                    where=rng.choice(["uniform", "mixed", "box"]), uvw=rng.random() < 0.5)
    if op == "grid":
        return dict(op="distance", mode="unsigned", mesh=rng.choice(["displaced", "tori"]),
                    level=rng.randint(3, 6), points=_log(rng, 32, 300) ** 3, where="grid", uvw=False)
    if op == "watertight":
        return dict(op="distance", mode="watertight", mesh=rng.choice(["icosphere", "displaced"]),
                    level=rng.randint(2, 6), points=_log(rng, 1000, 8 << 20),
                    where=rng.choice(["uniform", "mixed", "box"]), uvw=rng.random() < 0.25)
    if op == "raystab":
        return dict(op="distance", mode="raystab", mesh=rng.choice(["icosphere", "displaced"]),
                    level=rng.randint(2, 6), points=_log(rng, 1000, 3 << 20), where="box",
                    uvw=rng.random() < 0.25)
    if op == "camera":
        return dict(op="rays", kind="camera", level=rng.randint(2, 6), poses=rng.randint(1, 8),
                    width=_log(rng, 40, 2048), height=_log(rng, 40, 2048))
    if op == "random":
        return dict(op="rays", kind="random", level=rng.randint(2, 6), poses=1, width=_log(rng, 1000, 16 << 20),
                    height=1)
    if op == "gradient":
        return dict(op="gradient", mode=rng.choice(["unsigned", "watertight"]), level=rng.randint(2, 6),
                    points=_log(rng, 2000, 4 << 20))
    if op == "arena":
        return dict(op="arena", meshes=rng.randint(4, 48), max_level=rng.randint(3, 6), min_points=1000,
                    max_points=_log(rng, 5000, 200000))
    if op in ("floodfill", "udf_to_sdf"):
        if rng.random() < 0.5:   # a cube
            n = _log(rng, 32, 512)
            return dict(op=op, b=1, h=n, w=n, d=n)
        return dict(op=op, b=rng.randint(1, 4), h=rng.randint(20, 300), w=rng.randint(20, 300),
                    d=rng.randint(20, 300))
    return dict(op="marching_cubes", res=_log(rng, 24, 256), average=rng.random() < 0.5)


# ------------------------------------------------------------------ meshes
def _mesh(kind, level, seed):
    if kind == "icosphere":
        return W.icosphere(level, 0.8)
    if kind == "displaced":
        return W.displaced_icosphere(level, seed)
    return W.random_tori(seed)   # 12 open tori, about 177,000 faces


def _n_faces(kind, level):
    return 20 * 4 ** level if kind in ("icosphere", "displaced") else 176948


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(shape, g, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32) * (hi - lo) + lo


def _surface(v, f, n, band, g):
    """n points on area-weighted random faces, moved along the normal by U(-band, band)."""
    v = torch.as_tensor(v, device=DEV).double()
    f = torch.as_tensor(f, device=DEV)
    a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    nrm = torch.linalg.cross(b - a, c - a)
    area = nrm.norm(dim=1)
    cum = area.cumsum(0)
    r = _rand((4, n), g).double()
    k = torch.searchsorted(cum, r[0] * cum[-1]).clamp_(max=len(f) - 1)
    s = r[1].sqrt()
    w0, w1, w2 = 1 - s, s * (1 - r[2]), s * r[2]
    p = w0[:, None] * a[k] + w1[:, None] * b[k] + w2[:, None] * c[k]
    return (p + nrm[k] / area[k, None] * ((2 * r[3] - 1) * band)[:, None]).float()


def _points(where, n, v, f, g):
    if where == "uniform":
        return _rand((n, 3), g, -1, 1)
    if where == "mixed":
        h = n // 2
        return torch.cat([_rand((h, 3), g, -1, 1), _surface(v, f, n - h, 0.02, g)])
    if where == "box":
        lo, hi = torch.as_tensor(v.min(0), device=DEV), torch.as_tensor(v.max(0), device=DEV)
        return (lo + hi) / 2 + _rand((n, 3), g, -1, 1) * ((hi - lo) / 2 * 1.1)
    res = round(n ** (1 / 3))
    x = torch.linspace(-1, 1, res, device=DEV)
    return torch.stack(torch.meshgrid(x, x, x, indexing="ij"), -1).view(-1, 3)


def _cameras(poses, width, height, g):
    """Pinhole cameras (fov 50 degrees over the height) on the sphere of radius 2.5 looking at the origin."""
    c = torch.randn((poses, 3), generator=g, device=DEV, dtype=torch.float64)
    c = c / c.norm(dim=1, keepdim=True) * 2.5
    focal = height / 2 / math.tan(math.radians(25.0))
    y, x = torch.meshgrid(torch.arange(height, device=DEV, dtype=torch.float64),
                          torch.arange(width, device=DEV, dtype=torch.float64), indexing="ij")
    pix = torch.stack([(x + 0.5 - width / 2) / focal, -(y + 0.5 - height / 2) / focal, -torch.ones_like(x)], -1)
    pix = pix.view(-1, 3)
    os_, ds = [], []
    for k in range(poses):
        fwd = -c[k] / c[k].norm()
        up = torch.tensor([0.0, 1.0, 0.0] if abs(float(fwd[1])) < 0.99 else [1.0, 0.0, 0.0], device=DEV,
                          dtype=torch.float64)
        right = torch.linalg.cross(fwd, up)
        right = right / right.norm()
        rot = torch.stack([right, torch.linalg.cross(right, fwd), -fwd], 1)
        d = pix @ rot.T
        ds.append((d / d.norm(dim=1, keepdim=True)).float())
        os_.append(c[k].float().expand(len(pix), 3))
    return torch.cat(os_).contiguous(), torch.cat(ds).contiguous()


def _random_rays(n, g):
    """Half from anywhere in the box in any direction, half from outside towards the middle."""
    h = n // 2
    o1 = _rand((h, 3), g, -1, 1)
    d1 = torch.randn((h, 3), generator=g, device=DEV)
    s = torch.randn((n - h, 3), generator=g, device=DEV)
    o2 = 3 * s / s.norm(dim=1, keepdim=True)
    d2 = _rand((n - h, 3), g, -0.8, 0.8) - o2
    d = torch.cat([d1, d2])
    return torch.cat([o1, o2]).contiguous(), (d / d.norm(dim=1, keepdim=True)).contiguous()


def _tori_field(shape, seed):
    """Distance to the surfaces of eight tori at the voxels of [-1, 1]^3 (float32 [B, H, W, D]); a wedge is cut out
    of every second torus, so the free space inside it joins the outside."""
    B, H, Wd, D = shape
    out = torch.empty(shape, device=DEV)
    ax = [torch.linspace(-1, 1, n, device=DEV) for n in (H, Wd, D)]
    for b in range(B):
        rng = np.random.default_rng([seed, b])
        tori = []
        for _ in range(8):
            q, _r = np.linalg.qr(rng.standard_normal((3, 3)))
            tori.append((q.tolist(), rng.uniform(-0.5, 0.5, 3).tolist(), rng.uniform(0.2, 0.4), rng.uniform(0.08, 0.15)))
        for h0 in range(0, H, 64):   # a slab at a time
            x, y, z = ax[0][h0:h0 + 64, None, None], ax[1][None, :, None], ax[2][None, None, :]
            best = None
            for k, (q, c, R, r) in enumerate(tori):
                px, py, pz = x - c[0], y - c[1], z - c[2]
                u = q[0][0] * px + q[0][1] * py + q[0][2] * pz
                v = q[1][0] * px + q[1][1] * py + q[1][2] * pz
                w = q[2][0] * px + q[2][1] * py + q[2][2] * pz
                d = (((u * u + v * v).sqrt() - R) ** 2 + w * w).sqrt().sub_(r).abs_()
                if k % 2:
                    d = torch.where((u > 0) & (v.abs() < 0.2 * u), d + 0.2, d)
                best = d if best is None else torch.minimum(best, d)
            out[b, h0:h0 + 64] = best
    return out


_CORNERS = [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]]


def _band(res, seed):
    """Voxels of a band around a sphere of radius 0.418 res and a distance field at their corners: the signed
    distance to the sphere times a smooth positive factor that the seed draws."""
    rng = np.random.default_rng(seed)
    c = torch.tensor([res / 2 + 0.3, res / 2 - 0.2, res / 2 + 0.1], device=DEV, dtype=torch.float64)
    wave = torch.tensor(rng.uniform(-1, 1, 3), device=DEV)
    r = 0.418 * res
    i = torch.arange(res, device=DEV, dtype=torch.int32)
    g = torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).view(-1, 3)
    g = g[((g + 0.5 - c.float()).norm(dim=1) - r).abs() < 2.5].contiguous()
    at = (g[:, None] + torch.tensor(_CORNERS, device=DEV, dtype=torch.int32)).double()
    d = ((at - c).norm(dim=2) - r) * (1 + 0.4 * torch.sin((at * wave).sum(2)))
    return g, d.float().contiguous()


def _arena_inputs(case, seed):
    """Meshes (displaced icospheres and tori), their queries and modes (unsigned and raystab in turn); sizes are the
    case's, vertices and points the seed's."""
    rng = np.random.default_rng([case["meshes"], case["max_level"], case["max_points"]])
    shape = np.random.default_rng(seed)
    g = _gen(seed)
    meshes, pts, modes = [], [], []
    for m in range(case["meshes"]):
        level = int(rng.integers(2, case["max_level"] + 1))
        if m % 2 == 0 or level > 5:
            v, f = W.displaced_icosphere(level, seed + m)
        else:
            k = int(round(math.sqrt(20 * 4 ** level / 8)))
            v, f = W.torus(shape.uniform(0.3, 0.6), shape.uniform(0.08, 0.25), 4 * k, k)
            v = v.astype(np.float32)
        n = int(math.exp(rng.uniform(math.log(case["min_points"]), math.log(case["max_points"]))))
        meshes.append((v, f))
        pts.append(_points("box", n, v, f, g))
        modes.append("unsigned" if (m // 2) % 2 == 0 else "raystab")
    return meshes, pts, modes


# -------------------------------------------------------------------- state
def _inputs(case, seed):
    """The inputs alone, without the library's handles."""
    g = _gen(seed)
    op = case["op"]
    if op == "distance":
        v, f = _mesh(case["mesh"], case["level"], seed)
        return dict(v=v, f=f, points=_points(case["where"], case["points"], v, f, g))
    if op == "rays":
        v, f = _mesh("displaced", case["level"], seed)
        o, d = (_cameras(case["poses"], case["width"], case["height"], g) if case["kind"] == "camera"
                else _random_rays(case["width"], g))
        return dict(v=v, f=f, o=o, d=d)
    if op == "gradient":
        v, f = _mesh("displaced", case["level"], seed)
        n = case["points"]
        pts = torch.cat([_rand((n // 2, 3), g, -1, 1), _surface(v, f, n - n // 2, 0.05, g)])
        delta = _rand((len(v), 3), g, -1e-3, 1e-3)
        return dict(v=v, f=f, points=pts, weights=_rand((n,), g), base=torch.from_numpy(v).to(DEV), delta=delta)
    if op == "arena":
        meshes, pts, modes = _arena_inputs(case, seed)
        return dict(meshes=meshes, counts=[len(p) for p in pts], modes=modes, points=torch.cat(pts),
                    weights=_rand((sum(len(p) for p in pts),), g))
    if op in ("floodfill", "udf_to_sdf"):
        shape = (case["b"], case["h"], case["w"], case["d"])
        udf = _tori_field(shape, seed)
        return dict(grid=udf < 2.0 / case["d"]) if op == "floodfill" else dict(udf=udf)
    coords, corners = _band(case["res"], seed)
    return dict(coords=coords, corners=corners)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["op"] in ("distance", "rays", "gradient"):
        s["bvh"] = cubvh.cuBVH(s["v"], s["f"])
    if case["op"] == "gradient":
        s["points"].requires_grad_(True)
        s["delta"].requires_grad_(True)
    if case["op"] == "arena":
        s["arena"] = cubvh.BVHArena(s["meshes"])
        s["arena"].set_queries(s["counts"], s["modes"])
        s["points"].requires_grad_(True)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "distance":
        if case["mode"] == "unsigned":
            d, face, uvw = s["bvh"].unsigned_distance(s["points"], return_uvw=case["uvw"])
        else:
            d, face, uvw = s["bvh"].signed_distance(s["points"], return_uvw=case["uvw"], mode=case["mode"])
        return (d, face, uvw) if case["uvw"] else (d, face)
    if op == "rays":
        return s["bvh"].ray_trace(s["o"], s["d"])
    if op == "gradient":   # one fitting step: the vertices have moved, so the BVH is refitted
        vertices = s["base"] + s["delta"]
        if case["mode"] == "unsigned":
            d, face, _ = s["bvh"].unsigned_distance(s["points"], vertices=vertices)
        else:
            d, face, _ = s["bvh"].signed_distance(s["points"], mode=case["mode"], vertices=vertices)
        gp, gv = torch.autograd.grad((s["weights"] * d).sum(), [s["points"], s["delta"]])
        return d.detach(), face, gp, gv
    if op == "arena":
        d, face, _ = s["arena"].distance(s["points"])
        gp, = torch.autograd.grad((s["weights"] * d).sum(), [s["points"]])
        return d.detach(), face, gp
    if op == "floodfill":
        return cubvh.floodfill(s["grid"])
    if op == "udf_to_sdf":
        return cubvh.udf_to_sdf(s["udf"])
    return cubvh.sparse_marching_cubes(s["coords"], s["corners"], 0.0, ensure_consistency=case["average"])


# --------------------------------------------------------------------- work
def _walk_flops(faces):
    """One root-to-leaf path of an 8-wide tree (12 operations a box), a leaf of four triangles (100 each)."""
    return 8 * 12 * max(1.0, math.log(faces / 4, 8)) + 400


def work(case):
    op = case["op"]
    if op == "distance":
        n = case["points"]
        F = _n_faces(case["mesh"], case["level"])
        flops = n * _walk_flops(F)
        if case["mode"] == "raystab":   # a closed shape fills about a third of its box: those points need 64 rays
            flops += n * _walk_flops(F) * (2 + 0.33 * 62)
        return dict(bytes=n * (24 + (12 if case["uvw"] else 0)) + 18 * F, flops=flops)
    if op == "rays":
        n = case["poses"] * case["width"] * case["height"]
        F = _n_faces("displaced", case["level"])
        return dict(bytes=48 * n + 18 * F, flops=n * _walk_flops(F))
    if op == "gradient":
        n = case["points"]
        F = _n_faces("displaced", case["level"])
        # points, distance, face, weight, point gradient; mesh and vertex gradients
        return dict(bytes=n * (12 + 4 + 8 + 4 + 12) + F * (18 + 12), flops=n * (_walk_flops(F) + 100))
    if op == "arena":
        rng = np.random.default_rng(0)
        n = case["meshes"] * float(np.exp(rng.uniform(math.log(case["min_points"]), math.log(case["max_points"]),
                                                      4096)).mean())
        F = 20 * 4 ** ((2 + case["max_level"]) / 2)
        return dict(bytes=n * 40 + case["meshes"] * 18 * F,
                    flops=n * _walk_flops(F) * (1 + 0.5 * (2 + 0.2 * 62)))
    vox = 1
    if op in ("floodfill", "udf_to_sdf"):
        vox = case["b"] * case["h"] * case["w"] * case["d"]
        return dict(bytes=vox * (5 if op == "floodfill" else 8), flops=vox)
    n = 5 * 4 * math.pi * (0.418 * case["res"]) ** 2    # voxels of the band; about two vertices in five voxels
    return dict(bytes=n * (12 + 32) + 0.3 * n * 12 + 0.6 * n * 12, flops=60 * n)


# -------------------------------------------------------------------- exact
def _chunks(n, faces, elems=1 << 24):
    c = max(1, elems // max(faces, 1))
    return [(i, min(i + c, n)) for i in range(0, n, c)]


class _Faces:
    """Per-face tables for the squared distances of points to all faces (64 bits, by matrix products)."""

    def __init__(self, v, f):
        v = torch.as_tensor(v, device=DEV).double()
        f = torch.as_tensor(f, device=DEV)
        self.p = [v[f[:, k]] for k in range(3)]
        n = torch.linalg.cross(self.p[1] - self.p[0], self.p[2] - self.p[0])
        self.n = n / n.norm(dim=1, keepdim=True)
        self.e = [self.p[(k + 1) % 3] - self.p[k] for k in range(3)]
        self.out = [torch.linalg.cross(self.e[k], self.n) for k in range(3)]   # points out of the face

    def d2(self, x):
        xx = (x * x).sum(1, keepdim=True)
        best = inside = None
        for k in range(3):
            p, e = self.p[k], self.e[k]
            w2 = xx - 2 * (x @ p.T) + (p * p).sum(1)
            we = x @ e.T - (p * e).sum(1)
            ee = (e * e).sum(1)
            t = (we / ee).clamp_(0, 1)
            d = w2 - 2 * t * we + t * t * ee
            best = d if best is None else torch.minimum(best, d)
            s = (x @ self.out[k].T - (p * self.out[k]).sum(1)) <= 0
            inside = s if inside is None else inside & s
        h = x @ self.n.T - (self.p[0] * self.n).sum(1)
        return torch.where(inside, h * h, best).clamp_(min=0)

    def closest(self, x, k):
        """Closest point of face k[i] to x[i], and its barycentric weights."""
        P = [q[k] for q in self.p]
        cand, bary, ds = [], [], []
        for j in range(3):
            a, b = P[j], P[(j + 1) % 3]
            t = (((x - a) * (b - a)).sum(1) / ((b - a) ** 2).sum(1)).clamp(0, 1)
            c = a + t[:, None] * (b - a)
            w = torch.zeros_like(x)
            w[:, j], w[:, (j + 1) % 3] = 1 - t, t
            cand.append(c), bary.append(w), ds.append(((x - c) ** 2).sum(1))
        n = self.n[k]
        h = ((x - P[0]) * n).sum(1, keepdim=True)
        c = x - h * n
        area = ((torch.linalg.cross(P[1] - P[0], P[2] - P[0])) * n).sum(1)
        w = torch.stack([(torch.linalg.cross(P[(j + 2) % 3] - P[(j + 1) % 3], c - P[(j + 1) % 3]) * n).sum(1) / area
                         for j in range(3)], 1)
        inside = (w >= 0).all(1)
        cand.append(c), bary.append(w)
        ds.append(torch.where(inside, h[:, 0] ** 2, torch.full_like(h[:, 0], math.inf)))
        pick = torch.stack(ds, 1).argmin(1)
        i = torch.arange(len(x), device=DEV)
        return torch.stack(cand, 1)[i, pick], torch.stack(bary, 1)[i, pick]

    def near_normals(self, c):
        """Sum of the unit normals of the faces within 1e-3 of c."""
        return (self.d2(c) < 1e-6).double() @ self.n

    def winding(self, x):
        """Solid angle of the mesh seen from x over 4 pi."""
        a, b, c = self.p
        xx = (x * x).sum(1, keepdim=True)
        la, lb, lc = [(xx - 2 * (x @ q.T) + (q * q).sum(1)).clamp_(min=0).sqrt_() for q in self.p]

        def dot(p, q):
            return (p * q).sum(1) - x @ (p + q).T + xx

        num = (a * torch.linalg.cross(b, c)).sum(1) - x @ (torch.linalg.cross(a, b) + torch.linalg.cross(b, c)
                                                             + torch.linalg.cross(c, a)).T
        den = la * lb * lc + dot(a, b) * lc + dot(b, c) * la + dot(c, a) * lb
        return torch.atan2(num, den).sum(1) / (2 * math.pi)


def _distance64(v, f, x, mode):
    """(signed) distance, closest point, nearest face, barycentric weights."""
    faces = _Faces(v, f)
    x = x.detach().double()
    d, cp, face, bary = [], [], [], []
    for i, j in _chunks(len(x), len(f)):
        p = x[i:j]
        k = faces.d2(p).argmin(1)
        c, w = faces.closest(p, k)
        r = (p - c).norm(dim=1)
        if mode == "watertight":
            r = torch.where((faces.near_normals(c) * (p - c)).sum(1) < 0, -r, r)
        elif mode == "raystab":
            r = torch.where(faces.winding(p).abs() > 0.5, -r, r)
        d.append(r), cp.append(c), face.append(k), bary.append(w)
    return torch.cat(d), torch.cat(cp), torch.cat(face), torch.cat(bary)


def _rays64(v, f, o, d):
    v = torch.as_tensor(v, device=DEV).double()
    f = torch.as_tensor(f, device=DEV)
    a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    e1, e2 = b - a, c - a
    n = torch.linalg.cross(e1, e2)
    o, d = o.double(), d.double()
    depth = torch.full((len(o),), 1000.0, device=DEV, dtype=torch.float64)
    for i, j in _chunks(len(o), len(f)):
        oo, dd = o[i:j], d[i:j]
        m = torch.linalg.cross(oo, dd)
        det = -(dd @ n.T)
        U = m @ e2.T - dd @ torch.linalg.cross(e2, a).T
        V = -(m @ e1.T) - dd @ torch.linalg.cross(a, e1).T
        T = oo @ n.T - (a * n).sum(1)
        s = det.sign()
        hit = (s != 0) & (U * s >= 0) & (V * s >= 0) & ((U + V) * s <= det * s) & (T * s >= 0)
        t = torch.where(hit, T / det, torch.full_like(T, math.inf))
        best, k = t.min(1)
        exact_t = ((a[k] - oo) * n[k]).sum(1) / (dd * n[k]).sum(1)
        depth[i:j] = torch.where(best < 1000.0, exact_t, torch.full_like(best, 1000.0))
    return o + depth[:, None] * d, depth


def _outside(free):
    """The component of voxel (0, 0, 0) of each volume (0 where it is occupied: then all that is occupied)."""
    B, D, H, Wd = free.shape
    seen = torch.zeros_like(free)
    seen[:, 0, 0, 0] = free[:, 0, 0, 0]
    for step in range(20 * (D + H + Wd)):
        before = int(seen.sum()) if step % 16 == 0 else -1
        for ax in (1, 2, 3):
            n = free.shape[ax]
            old = seen.clone()
            seen.narrow(ax, 0, n - 1).logical_or_(old.narrow(ax, 1, n - 1))
            seen.narrow(ax, 1, n - 1).logical_or_(old.narrow(ax, 0, n - 1))
            seen &= free
        if before >= 0 and int(seen.sum()) == before:
            break
    first_occupied = ~free[:, 0, 0, 0]
    return torch.where(first_occupied.view(-1, 1, 1, 1), ~free, seen)


def exact(case, seed):
    op = case["op"]
    if op == "distance":
        pairs = case["points"] * float(_n_faces(case["mesh"], case["level"]))
        if pairs * (1 if case["mode"] == "unsigned" else 2) > MAX_PAIRS:
            return None
        s = _inputs(case, seed)
        d = _distance64(s["v"], s["f"], s["points"], case["mode"])[0]
        return (d, None, None) if case["uvw"] else (d, None)   # nearest faces tie at edges, and uvw with them
    if op == "rays":
        n = case["poses"] * case["width"] * case["height"]
        if n * float(_n_faces("displaced", case["level"])) > MAX_PAIRS:
            return None
        s = _inputs(case, seed)
        pos, depth = _rays64(s["v"], s["f"], s["o"], s["d"])
        return pos, None, depth
    if op == "gradient":
        if case["points"] * float(_n_faces("displaced", case["level"])) * 2 > MAX_PAIRS:
            return None
        s = _inputs(case, seed)
        v = s["base"] + s["delta"]   # the mesh that the call is given (float32)
        f = torch.as_tensor(s["f"], device=DEV)
        d, cp, face, bary = _distance64(v, f, s["points"], case["mode"])
        g = s["weights"].double()[:, None] * (s["points"].double() - cp) / d[:, None]
        gv = torch.zeros(len(v), 3, device=DEV, dtype=torch.float64)
        for k in range(3):
            gv.index_add_(0, f[face, k], -bary[:, k:k + 1] * g)
        return d, None, g, gv
    if op == "arena":
        s = _inputs(case, seed)
        if sum(2.0 * len(m[1]) * c for m, c in zip(s["meshes"], s["counts"])) > MAX_PAIRS:
            return None
        ds, gs, at = [], [], 0
        for (v, f), n, mode in zip(s["meshes"], s["counts"], s["modes"]):
            p, w = s["points"][at:at + n], s["weights"][at:at + n]
            d, cp, _, _ = _distance64(v, f, p, mode)
            ds.append(d)
            gs.append(w.double()[:, None] * (p.double() - cp) / d[:, None])
            at += n
        return torch.cat(ds), None, torch.cat(gs)
    if op == "udf_to_sdf":
        udf = _inputs(case, seed)["udf"]
        eps = torch.tensor(2.0 / case["d"], dtype=torch.float32, device=DEV)
        # the fill's neighbourhood: a volume's memory as [D][H][W]
        free = ~(udf < eps).view(case["b"], case["d"], case["h"], case["w"])
        sdf = udf.double() - eps.double()
        inside = ~_outside(free).view(udf.shape)
        return torch.where(inside & (sdf > 0), -sdf, sdf)
    if op == "marching_cubes":
        s = _inputs(case, seed)
        g, val = s["coords"].long(), s["corners"].double()
        off = torch.tensor(_CORNERS, device=DEV)
        pairs = [(i, j) for i in range(8) for j in range(i + 1, 8)
                 if sum(abs(p - q) for p, q in zip(_CORNERS[i], _CORNERS[j])) == 1]
        size = case["res"] + 2
        keys, pos = [], []
        for i, j in pairs:
            axis = [p != q for p, q in zip(_CORNERS[i], _CORNERS[j])].index(True)
            if _CORNERS[i][axis] > _CORNERS[j][axis]:
                i, j = j, i
            cut = (val[:, i] < 0) != (val[:, j] < 0)
            a = g[cut] + off[i]
            t = -val[cut, i] / (val[cut, j] - val[cut, i])
            keys.append(((a[:, 0] * size + a[:, 1]) * size + a[:, 2]) * 3 + axis)
            pos.append(a.double() + t[:, None] * (off[j] - off[i]).double())
        keys, pos = torch.cat(keys), torch.cat(pos)
        key, inv = torch.unique(keys, return_inverse=True)
        out = torch.empty(len(key), 3, device=DEV, dtype=torch.float64)
        out[inv] = pos
        return out, None
    return None
