"""Timed cases of the SNCH-LBVH framework: what a walk-on-stars or geometry program
has it do, through the public Python calls.

``listed()`` names twelve calls over the range of use (a solver step on a small
mesh, rebuilds, each query type from small to full batches, batched meshes, a
whole walk, 2D scenes, learned radii); ``draw()`` gives further sizes of the
same kinds. A case's ``kind`` selects one entry of ``_KINDS`` below.

Meshes are the repository's synthetic ones: noisy icospheres (20 * 4^level
triangles), the 64-mesh scene of 1,993,600 triangles in the unit cube, batches
of icospheres and tori, and planar loops and open polylines. Every seed has its
own vertex noise and its own queries.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import snch_lbvh_gb300 as snch
from snch_lbvh_gb300 import meshes, wost
from snch_lbvh_gb300.learned import LearnedRadius

FULL = 1_993_600  # triangles of the 64-mesh scene


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # one step of a small interactive solver: the mesh moved, so rebuild, then a
        # few thousand queries of every type (launches and latency)
        {"name": "step_small", "kind": "step", "level": 3, "n": 4096},
        # a scene whose geometry changes every step: topology and tree of the full scene
        {"name": "build_full", "kind": "build", "level": -1},
        # closest-point queries against one scanned object: a dense ordinary batch
        {"name": "near_object", "kind": "near", "level": 5, "n": 1_000_000},
        # the distance query of a walk-on-stars step on the full scene, largest batch
        {"name": "near_full", "kind": "near", "level": -1, "n": 16_000_000},
        # silhouette queries late in a walk: a few walkers are left, an odd count
        {"name": "sil_few", "kind": "sil", "level": 5, "n": 20_011},
        # the silhouette query of a walk-on-stars step on the full scene, largest batch
        {"name": "sil_full", "kind": "sil", "level": -1, "n": 16_000_000},
        # the ray query of the same step, largest batch
        {"name": "ray_full", "kind": "ray", "level": -1, "n": 16_000_000},
        # its boundary samples: a draw in a sphere, then a point on the drawn triangle
        {"name": "sample_full", "kind": "sample", "level": -1, "n": 4_000_000},
        # many independent objects served together: nearest and silhouette batches
        {"name": "batch_meshes", "kind": "batch", "meshes": 24, "hi": 50_000, "per_tri": 8},
        # a whole walk-on-stars solve, its batches shrinking as walkers end
        {"name": "walk_solve", "kind": "walk", "level": 5, "walkers": 100_003, "steps": 64},
        # a planar scene: the four 2D queries
        {"name": "flat_scene", "kind": "flat", "loops": 400, "n": 200_000},
        # search radii from the learned model, then the searches they seed
        {"name": "learned_full", "kind": "learned", "level": -1, "n": 4_000_000},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "build", "near", "near", "sil", "sil", "ray", "sample", "batch", "walk", "flat",
                       "learned"])
    if kind == "step":
        return {"kind": kind, "level": rng.randint(2, 5), "n": size(1_000, 60_000)}
    if kind == "build":
        return {"kind": kind, "level": -2, "quads": size(100, 1_000_000)}
    if kind in ("near", "sil", "ray", "sample", "learned"):
        level = rng.choice([3, 4, 5, 6, -1, -1])
        top = {"near": 16_000_000, "sil": 16_000_000, "ray": 16_000_000, "sample": 4_000_000,
               "learned": 4_000_000}[kind]
        if level >= 0:  # inside a closed mesh a silhouette search visits much of it
            top = 400_000 if kind in ("sil", "learned") else 4_000_000
        return {"kind": kind, "level": level, "n": size(2_000, top)}
    if kind == "batch":
        return {"kind": kind, "meshes": rng.randint(2, 24), "hi": size(4_000, 50_000), "per_tri": rng.randint(1, 8)}
    if kind == "walk":
        return {"kind": kind, "level": rng.randint(3, 5), "walkers": size(5_000, 100_000),
                "steps": rng.randint(16, 64)}
    return {"kind": kind, "loops": size(4, 400), "n": size(2_000, 200_000)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _log_uniform(g, n, lo, hi):
    return torch.exp(math.log(lo) + (math.log(hi) - math.log(lo)) * _rand(g, n))


def _directions(g, n, dim):
    d = torch.randn(n, dim, generator=g, device="cuda")
    return d / d.norm(dim=1, keepdim=True)


@functools.lru_cache(maxsize=None)
def _sphere(level):
    v, f, _ = meshes.icosphere(level)
    return torch.from_numpy(v.astype(np.float32)), torch.from_numpy(f)


@functools.lru_cache(maxsize=None)
def _full():
    s = meshes.wost_scene()
    return torch.from_numpy(s.verts), torch.from_numpy(s.faces)


@functools.lru_cache(maxsize=None)
def _batch(count, hi):
    return [(torch.from_numpy(v), torch.from_numpy(f))
            for v, f in meshes.batched_meshes(seed=5, count=count, lo=1e3, hi=hi)]


def _torus_sides(quads):
    nu = max(6, int(math.sqrt(2 * quads)))
    return nu, max(3, quads // nu)


def _mesh(level, g, quads=0):
    """Vertices and triangles on the GPU. level >= 0: an icosphere of radius 1 with 1 % noise
    along its normals; -1: the 64-mesh scene, its vertices moved by 0.01 % of the cube; -2: a
    torus of about `quads` quads, two triangles each, moved likewise."""
    if level == -2:
        nu, nv = _torus_sides(quads)
        v, f = meshes.torus(0.35, 0.1, nu, nv)[:2]
        v, f = torch.from_numpy(v.astype(np.float32)).cuda(), torch.from_numpy(f).cuda()
        return v + 1e-4 * torch.randn(v.shape, generator=g, device="cuda"), f
    if level >= 0:
        v, f = _sphere(level)
        v, f = v.cuda(), f.cuda()
        return v * (1.0 + 0.01 * torch.randn(len(v), 1, generator=g, device="cuda")), f
    v, f = _full()
    v, f = v.cuda(), f.cuda()
    return v + 1e-4 * torch.randn(v.shape, generator=g, device="cuda"), f


def _points(level, n, g):
    """Query points: uniform in the sphere's box x 1.2, or in the unit cube."""
    p = _rand(g, n, 3)
    return (2.0 * p - 1.0) * 1.2 if level >= 0 else p


def _scale(level):
    return 2.0 if level >= 0 else 1.0


def _rays(level, n, g):
    return _points(level, n, g), _directions(g, n, 3), _log_uniform(g, n, 1e-3, 1.0) * _scale(level)


def _draws(level, n, g):
    return _points(level, n, g), _log_uniform(g, n, 1e-3, 0.5) * _scale(level), _rand(g, n)


def _flips(n, g):
    return (_rand(g, n) < 0.5).to(torch.uint8)


def _built(v, f):
    s = snch.Scene(v, f)
    s.compute_silhouettes()
    s.build_bvh()
    return s


def _device_array(ptr, rows, cols, typestr):
    class _Mem:
        __cuda_array_interface__ = {"shape": (rows, cols), "typestr": typestr, "data": (int(ptr), False),
                                    "version": 3}

    return torch.as_tensor(_Mem(), device="cuda")


def _tree(scene):
    """The built tree as the device-side view gives it: nodes, boxes, normal cones."""
    b = scene.get_bvh_device_ptr()
    return (_device_array(b.nodes, b.num_nodes, 4, "<i4"), _device_array(b.aabbs, b.num_nodes, 6, "<f4"),
            _device_array(b.cones, b.num_nodes, 5, "<f4"))


def _polylines(loops, seed):
    """Noisy closed loops and, every third one, open polylines of 8 to 900 segments, in a
    20 x 20 square (smaller for few loops, so that the density stays)."""
    rng = np.random.default_rng(seed)
    side = math.sqrt(loops)
    verts, segs, off = [], [], 0
    for k in range(loops):
        m = int(rng.integers(8, 900))
        c = rng.random(2) * side
        a = np.sort(rng.random(m)) * 2 * np.pi
        r = rng.uniform(0.05, 0.6) * (1 + 0.02 * rng.standard_normal(m))
        verts.append(np.stack([c[0] + r * np.cos(a), c[1] + r * np.sin(a)], 1))
        i = np.arange(m)
        segs.append(np.stack([i, (i + 1) % m], 1)[: m if k % 3 else m - 1] + off)
        off += m
    return np.concatenate(verts).astype(np.float32), np.concatenate(segs).astype(np.int32), side


def _model_layers(seed):
    """Weights and biases of the radius model's five layers: He-uniform hidden layers and a
    small head around log 0.05, about the median distance in the unit cube."""
    rng = np.random.default_rng(seed)
    out = []
    for i, (k, m) in enumerate([(192, 64), (64, 64), (64, 64), (64, 64), (64, 2)]):
        b = math.sqrt(6.0 / k) if i < 4 else 0.1 * math.sqrt(3.0 / k)
        out.append((rng.uniform(-b, b, (m, k)).astype(np.float32),
                    np.full(m, 0.0 if i < 4 else math.log(0.05), np.float32)))
    return out


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        parts, mesh, pts = [], [], {"near": [], "sil": []}
        for k, (v, f) in enumerate(_batch(case["meshes"], float(case["hi"]))):
            v = v.cuda() + 1e-4 * torch.randn(v.shape, generator=g, device="cuda")
            parts.append((v, f.cuda()))
            lo, hi = v.min(0).values, v.max(0).values
            c, h = 0.5 * (lo + hi), 0.6 * (hi - lo)
            n = case["per_tri"] * len(f)
            mesh.append(torch.full((n,), k, dtype=torch.int32, device="cuda"))
            for p in pts.values():
                p.append(c + (2.0 * _rand(g, n, 3) - 1.0) * h)
        s = snch.BatchedScene(parts)
        s.compute_silhouettes()
        s.build_bvh()
        return {"kind": kind, "scene": s, "mesh": torch.cat(mesh), "near": torch.cat(pts["near"]),
                "sil": torch.cat(pts["sil"])}
    if kind == "flat":
        v, segs, side = _polylines(case["loops"], seed)
        s = snch.Scene2(v, segs)
        s.build()
        n = case["n"]
        p = _rand(g, n, 2) * (side + 1.0) - 0.5
        return {"kind": kind, "scene": s, "p": p, "flip": _flips(n, g), "d": _directions(g, n, 2),
                "tmax": _log_uniform(g, n, 1e-2, 30.0), "r": _log_uniform(g, n, 1e-2, 3.0), "u": _rand(g, n)}
    if kind == "walk":
        v, f = _mesh(case["level"], g)
        neumann = (_rand(g, len(f)) < 0.5).cpu().numpy()
        d, nm = wost.split_boundary(v.cpu().numpy(), f.cpu().numpy(), neumann)
        return {"kind": kind, "d": d, "n": nm, "walkers": case["walkers"], "steps": case["steps"], "seed": seed}
    v, f = _mesh(case["level"], g, case.get("quads", 0))
    s = _built(v, f)
    st = {"kind": kind, "scene": s}
    if kind == "build":
        return st
    n, level = case["n"], case["level"]
    if kind in ("near", "sil", "step", "learned"):
        st["p"] = _points(level, n, g)
    if kind in ("sil", "step"):
        st["flip"] = _flips(n, g)
    if kind in ("ray", "step"):
        st["ray"] = _rays(level, n, g)
    if kind in ("sample", "step"):
        st["draw"] = _draws(level, n, g)
        st["uv"] = (_rand(g, n), _rand(g, n))
    if kind == "learned":
        half = 1.2 if level >= 0 else 1.0
        lo = -half if level >= 0 else 0.0
        m = LearnedRadius(np.full(3, lo), np.full(3, half), seed=0)
        m.params = np.concatenate([x.reshape(-1) for w, b in _model_layers(seed) for x in (w, b)])
        st["model"], st["margin"] = m, 1.5 * _scale(level)
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    kind = st["kind"]
    if kind == "flat":
        s = st["scene"]
        return (s.query_nearest(st["p"]), s.query_silhouette(st["p"], st["flip"]),
                s.query_ray(st["p"], st["d"], st["tmax"]), s.sample_in_circle(st["p"], st["r"], st["u"]))
    if kind == "walk":
        est, start, _ = wost.trace(st["d"], st["n"], st["walkers"], max_steps=st["steps"], seed=st["seed"])
        return est, start
    s = st["scene"]
    if kind == "build":
        s.compute_silhouettes()
        s.build_bvh()
        return _tree(s)
    if kind == "near":
        return s.query_nearest(st["p"])
    if kind == "sil":
        return s.query_silhouette(st["p"], st["flip"])
    if kind == "ray":
        return s.query_ray(*st["ray"])
    if kind == "sample":
        idx, pdf = s.sample_in_sphere(*st["draw"])
        return idx, pdf, s.sample_on_object(idx.clamp(min=0), *st["uv"])
    if kind == "batch":
        return s.query_nearest_batch(st["mesh"], st["near"]), s.query_silhouette_batch(st["mesh"], st["sil"])
    if kind == "learned":
        rn, rs = st["model"].predict(st["p"], margin=st["margin"])
        return (rn, rs), s.query_nearest_seeded(st["p"], rn), s.query_silhouette_seeded(st["p"], rs)
    s.build_bvh()
    return (s.query_nearest(st["p"]), s.query_silhouette(st["p"], st["flip"]), s.query_ray(*st["ray"]),
            s.sample_in_sphere(*st["draw"]))


# ------------------------------------------------------------------ the work of a pass
def _tris(case):
    if case["kind"] == "batch":
        return sum(len(f) for _, f in _batch(case["meshes"], float(case["hi"])))
    if case["level"] == -2:
        nu, nv = _torus_sides(case["quads"])
        return 2 * nu * nv
    return FULL if case["level"] < 0 else 20 * 4 ** case["level"]


def _build_bytes(t):
    # vertices and triangles in; nodes, boxes and cones of 2t - 1 nodes out
    return 6 * t + 12 * t + 2 * t * (16 + 24 + 20)


def work(case):
    """Bytes: each input and output once and the geometry once (vertices, triangles; boxes,
    and for silhouettes cones, of the tree). Operations: one root-to-leaf path per query,
    two child tests a level and one element test at its end."""
    kind = case["kind"]
    if kind == "flat":
        t, n = 450 * case["loops"], case["n"]
        return {"bytes": t * (16 + 2 * 32) + n * (4 * 16 + 40 + 33), "flops": n * 4 * (2 * 12 * math.log2(t) + 30)}
    t = _tris(case)
    depth = math.log2(max(t, 2))
    box, cone, tri = 20.0, 30.0, 60.0  # operations of a box, a cone and an element test
    near, sil = depth * 2 * box + tri, depth * 2 * (box + cone) + tri
    geo, cones = 18 * t + 2 * t * 24, 2 * t * 20
    if kind == "build":
        return {"bytes": _build_bytes(t), "flops": 300 * t}
    if kind == "walk":  # half of the walkers are live at a typical step
        n = case["walkers"] * case["steps"] // 2
        return {"bytes": geo + cones + 16 * case["walkers"] + n * 60, "flops": n * (3 * near + sil)}
    if kind == "batch":
        n = case["per_tri"] * t
        return {"bytes": geo + cones + n * 2 * (16 + 8), "flops": n * (near + sil)}
    n = case["n"]
    if kind == "near":
        return {"bytes": geo + n * (12 + 8), "flops": n * near}
    if kind == "sil":
        return {"bytes": geo + cones + n * (13 + 8), "flops": n * sil}
    if kind == "ray":
        return {"bytes": geo + n * (28 + 17), "flops": n * near}
    if kind == "sample":
        return {"bytes": geo + n * (20 + 8 + 8 + 12), "flops": n * near}
    if kind == "learned":
        return {"bytes": geo + cones + n * (12 + 8 + 16), "flops": n * (2 * 24_576 + near + sil)}
    return {"bytes": _build_bytes(t) + n * (12 + 8 + 13 + 8 + 28 + 17 + 20 + 8),
            "flops": 300 * t + n * (3 * near + sil)}


# ------------------------------------------------------------------ 64-bit values
def _segment_sq(p, a, b):
    u = b - a
    s = (((p - a) * u).sum(-1) / (u * u).sum(-1).clamp(min=1e-300)).clamp(0.0, 1.0)
    return ((p - a - s.unsqueeze(-1) * u) ** 2).sum(-1)


def _triangle_sq(p, a, b, c):
    ab, ac, ap = b - a, c - a, p - a
    n = torch.linalg.cross(ab, ac)
    nn = (n * n).sum(-1)
    w = (torch.linalg.cross(ab, ap) * n).sum(-1)
    v = (torch.linalg.cross(ap, ac) * n).sum(-1)
    inside = (v >= 0) & (w >= 0) & (v + w <= nn) & (nn > 0)
    plane = (ap * n).sum(-1) ** 2 / nn.clamp(min=1e-300)
    edge = torch.minimum(_segment_sq(p, a, b), torch.minimum(_segment_sq(p, b, c), _segment_sq(p, c, a)))
    return torch.where(inside, plane, edge)


def _spheres(corners):
    """Centre and radius (32 bits, a little too large) of each element's bounding sphere."""
    centre = sum(corners) / len(corners)
    radius = torch.stack([(c - centre).norm(dim=1) for c in corners]).amax(0)
    return centre.float(), radius.float() * 1.0001 + 1e-4


def _nearest_distance(points, corners):
    """Distance of each point to the nearest of the elements (corners: 2 or 3 tensors of
    vertices). The element whose bounding sphere is nearest gives an upper bound; every
    element whose sphere is nearer than that is measured."""
    points, corners = points.double(), [c.double() for c in corners]
    sq = _segment_sq if len(corners) == 2 else _triangle_sq
    centre, radius = _spheres(corners)
    out = []
    for p in points.split(max(1, 400_000_000 // len(centre))):
        f = p.float()
        low = sum((f[:, k:k + 1] - centre[:, k]) ** 2 for k in range(f.shape[1])).sqrt_().sub_(radius)
        first = low.argmin(1)
        best = sq(p, *[c[first] for c in corners])
        i, j = torch.nonzero(low < (best.sqrt().float() * 1.0001 + 1e-4).unsqueeze(1), as_tuple=True)
        for a, b in zip(i.split(20_000_000), j.split(20_000_000)):
            best.scatter_reduce_(0, a, sq(p[a], *[c[b] for c in corners]), "amin")
        out.append(best.sqrt())
    return torch.cat(out)


def _first_hit(o, d, tmax, corners):
    """(hit, t) of the closest intersection with triangles or segments below tmax: every
    element whose bounding sphere the ray's line meets is tested."""
    o, d, tmax, corners = o.double(), d.double(), tmax.double(), [c.double() for c in corners]
    centre, radius = _spheres(corners)
    e1 = corners[1] - corners[0]
    rows = max(1, 200_000_000 // len(centre))
    out = []
    for po, pd, pm in zip(o.split(rows), d.split(rows), tmax.split(rows)):
        fo, fd = po.float(), pd.float()
        v = [centre[:, k] - fo[:, k:k + 1] for k in range(fo.shape[1])]
        if len(v) == 2:
            off = (v[0] * fd[:, 1:] - v[1] * fd[:, :1]) ** 2
        else:
            off = sum((v[a] * fd[:, b:b + 1] - v[b] * fd[:, a:a + 1]) ** 2 for a, b in ((0, 1), (1, 2), (2, 0)))
        i, j = torch.nonzero(off <= (radius * 1.001) ** 2, as_tuple=True)
        so, dd, f1 = po[i] - corners[0][j], pd[i], e1[j]
        if len(corners) == 3:
            f2 = corners[2][j] - corners[0][j]
            h = torch.linalg.cross(dd, f2)
            det = (f1 * h).sum(-1)
            u = (so * h).sum(-1) / det
            q = torch.linalg.cross(so, f1)
            w = (dd * q).sum(-1) / det
            t = (f2 * q).sum(-1) / det
            ok = (u >= 0) & (w >= 0) & (u + w <= 1)
        else:
            det = dd[:, 1] * f1[:, 0] - dd[:, 0] * f1[:, 1]
            t = (so[:, 0] * f1[:, 1] - so[:, 1] * f1[:, 0]) / det
            w = (dd[:, 1] * so[:, 0] - dd[:, 0] * so[:, 1]) / det
            ok = (w >= -1e-3) & (w <= 1 + 1e-3)
        t = torch.where(ok & (det != 0) & (t >= 0), t, torch.inf)
        first = torch.full((len(po),), torch.inf, dtype=torch.float64, device="cuda").scatter_reduce_(0, i, t, "amin")
        out.append(torch.where(first < pm, first, torch.inf))
    t = torch.cat(out)
    return (t < torch.inf).to(torch.uint8), t


def _radii(p, layers, lo, half, margin):
    """The radius model in 64 bits: Fourier features, four ReLU layers, two log radii."""
    u = ((p.double() - lo) / half - 1.0)
    s = torch.from_numpy(np.exp2(0.25 * np.arange(32)).astype(np.float32)).double().cuda()
    out = []
    for x in u.split(500_000):
        ph = math.pi * (s.view(32, 1) * x.unsqueeze(1))  # column 6 k + 2 a (+ 1): frequency k, axis a
        h = torch.stack([ph.sin(), ph.cos()], -1).reshape(len(x), 192)
        for i, (w, b) in enumerate(layers):
            h = h @ torch.from_numpy(w).double().cuda().T + torch.from_numpy(b).double().cuda()
            if i < 4:
                h = h.clamp(min=0)
        out.append(torch.exp(h) * margin)
    r = torch.cat(out)
    return r[:, 0], r[:, 1]


def exact(case, seed):
    """Distances, ray parameters and radii by brute force in 64 bits. The other outputs have
    no value apart from the tree and the traversal that give them: nodes and their boxes and
    cones, a silhouette distance (its cone test decides in 32 bits which edges are reached),
    a draw's triangle and density, a random walk's estimate, and which of several elements at
    the same distance is named."""
    kind = case["kind"]
    if kind == "flat":
        v, segs, _ = _polylines(case["loops"], seed)
        c = [torch.from_numpy(v[segs[:, k]]).cuda() for k in range(2)]
        g, n = _gen(seed), case["n"]
        p = _rand(g, n, 2) * (math.sqrt(case["loops"]) + 1.0) - 0.5
        _flips(n, g)
        d = _directions(g, n, 2)
        hit, t = _first_hit(p, d, _log_uniform(g, n, 1e-2, 30.0), c)
        return (None, _nearest_distance(p, c)), (None, None), (None, t, None, None), (None, None)
    if kind not in ("near", "step", "learned"):
        return None
    if kind == "learned" or (kind == "near" and case["level"] >= 0 and case["n"] * _tris(case) <= 2.1e10) or (
            kind == "step" and case["n"] * _tris(case) <= 5e8):
        g, n, level = _gen(seed), case["n"], case["level"]
        v, f = _mesh(level, g)
        p = _points(level, n, g)
        if kind == "learned":
            half = 1.2 if level >= 0 else 0.5
            r = _radii(p, _model_layers(seed), -1.2 if level >= 0 else 0.0, half, 1.5 * _scale(level))
            return r, (None, None), (None, None)
        c = [v[f[:, k].long()] for k in range(3)]
        near = (None, _nearest_distance(p, c))
        if kind == "near":
            return near
        _flips(n, g)
        hit, t = _first_hit(*_rays(level, n, g), c)
        return near, (None, None), (None, t, None, None), (None, None)
    return None
