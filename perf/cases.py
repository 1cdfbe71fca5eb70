"""The workloads this framework's speed is judged by: closest points, rays and silhouettes
on 3D meshes and 2D polylines, from one probe of a few points to millions of queries, and
mixed steps over many scenes.

A case names a family (`kind`), the geometry's size (`level`: subdivided icosahedron with
20 * 4^level triangles, displaced; `segs`: segments of a star polyline) and the number of
queries `n`.  The scenes are built once per process, as a program that queries a shape
many times does; the queries come from the seed.  Query points are uniform in the box
[-2, 2]^D the benchmark uses, or lie near the surface (`near`), as samples of a distance
field do.  `soa` arrays are [D, n] (the layout of the reference's arrays), the others
[n, D].
"""
from __future__ import annotations

import functools
import math

import torch

from gquery_b200 import Mesh, Polyline, Scene
from gquery_b200 import workloads as W
from gquery_b200.batch import SceneBatch

DEV = "cuda:0"
AMPLITUDE = {"cp3d": 0.15, "ray3d": 0.15, "sil3d": 0.3, "batch3d": 0.15}


def listed():
    return [
        # a program asking for the nearest surface point of a handful of probes: launches and latency
        {"name": "cp3d_probe", "kind": "cp3d", "level": 5, "n": 16, "near": False, "soa": True},
        # contact points of a few thousand particles against a detailed mesh
        {"name": "cp3d_few", "kind": "cp3d", "level": 7, "n": 2003, "near": False, "soa": False},
        # training samples of a distance field: points scattered about the surface
        {"name": "cp3d_near", "kind": "cp3d", "level": 7, "n": 250007, "near": True, "soa": True},
        # the benchmark's closest points: 8 M points over 1.3 M triangles
        {"name": "cp3d_large", "kind": "cp3d", "level": 8, "n": 8388608, "near": False, "soa": True},
        # visibility of a few thousand segments of limited length
        {"name": "ray3d_few", "kind": "ray3d", "level": 6, "n": 5003, "r_max": True, "soa": False},
        # the benchmark's rays
        {"name": "ray3d_large", "kind": "ray3d", "level": 8, "n": 8388608, "r_max": False, "soa": True},
        # a walk-on-stars step on a mesh: silhouettes of a moderate set of points
        {"name": "sil3d_some", "kind": "sil3d", "level": 6, "n": 30011, "r_max": False, "soa": False},
        # the benchmark's silhouettes
        {"name": "sil3d_large", "kind": "sil3d", "level": 7, "n": 4194304, "r_max": False, "soa": True},
        # the benchmark's closest points on a polyline
        {"name": "cp2d_large", "kind": "cp2d", "segs": 4096, "n": 1048576, "soa": True},
        # one walk-on-stars step in the plane: distance to the absorbing boundary, silhouettes
        # of the reflecting one within it, rays up to the star's radius
        {"name": "wost2d", "kind": "wost2d", "segs": 16384, "n": 65521, "soa": True},
        # one step over many uneven polylines, three kinds of queries in one launch
        {"name": "batch2d", "kind": "batch2d", "scenes": 48, "segs": 65536, "n": 1000003},
        # a small step over several meshes, in the forms the serving runtime launches
        {"name": "batch3d", "kind": "batch3d", "scenes": 8, "level": 6, "n": 24001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    case = _drawn(rng)
    if case["n"] < 4 and "soa" in case:
        case["soa"] = True  # a [n, D] array of D points would read as [D, n]
    return case


def _drawn(rng):
    kind = rng.choice(["cp3d", "cp3d", "ray3d", "sil3d", "cp2d", "wost2d", "batch2d", "batch3d"])
    soa = rng.random() < 0.5
    if kind == "cp3d":
        return {"kind": kind, "level": rng.randint(4, 8), "n": _log_int(rng, 1, 1 << 21), "near": rng.random() < 0.5,
                "soa": soa}
    if kind == "ray3d":
        return {"kind": kind, "level": rng.randint(4, 8), "n": _log_int(rng, 1, 1 << 23), "r_max": rng.random() < 0.5,
                "soa": soa}
    if kind == "sil3d":
        return {"kind": kind, "level": rng.randint(4, 7), "n": _log_int(rng, 1, 1 << 20), "r_max": rng.random() < 0.5,
                "soa": soa}
    if kind == "cp2d":
        return {"kind": kind, "segs": _log_int(rng, 64, 1 << 18), "n": _log_int(rng, 1, 1 << 22), "soa": soa}
    if kind == "wost2d":
        return {"kind": kind, "segs": _log_int(rng, 64, 1 << 17), "n": _log_int(rng, 1, 1 << 20), "soa": soa}
    if kind == "batch2d":
        return {"kind": kind, "scenes": rng.randint(2, 64), "segs": _log_int(rng, 1024, 1 << 16),
                "n": _log_int(rng, 1000, 1 << 21)}
    return {"kind": kind, "scenes": rng.randint(2, 10), "level": rng.randint(4, 6), "n": _log_int(rng, 300, 100000)}


# ---- scenes and inputs ---------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _mesh_data(level, amplitude, seed=0):
    v, f = W.icosphere(level, amplitude=amplitude, seed=seed)
    return torch.as_tensor(v), torch.as_tensor(f)


@functools.lru_cache(maxsize=None)
def _line_data(segs, seed=0, scale=1.0):
    v, e = W.star_polyline(segs, seed=seed)
    return torch.as_tensor(v) * scale, torch.as_tensor(e)


@functools.lru_cache(maxsize=None)
def _mesh(kind, level):
    v, f = _mesh_data(level, AMPLITUDE[kind])
    if kind == "sil3d":
        return Mesh(v.t(), f.t())
    return Scene(v, f, 3, build_snch=False)


@functools.lru_cache(maxsize=None)
def _line(segs, scale=1.0):
    v, e = _line_data(segs, 0, scale)
    return Polyline(v.t(), e.t())


def _uneven(scenes, segs):
    """Segment counts of a batch's polylines, evenly spread over their logarithm."""
    return [int(round(64 * (segs / 64) ** (k / (scenes - 1)))) for k in range(scenes)]


@functools.lru_cache(maxsize=None)
def _batch2d(scenes, segs):
    return [Scene(*_line_data(m, seed=k), 2) for k, m in enumerate(_uneven(scenes, segs))]


@functools.lru_cache(maxsize=None)
def _batch3d(scenes, level):
    return [Scene(*_mesh_data(3 + k % (level - 2), AMPLITUDE["batch3d"], seed=k), 3) for k in range(scenes)]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _box(n, dim, g):
    return torch.rand((n, dim), generator=g, device=DEV) * 4.0 - 2.0


def _dirs(n, dim, g):
    d = torch.randn((n, dim), generator=g, device=DEV, dtype=torch.float64)
    return (d / d.norm(dim=1, keepdim=True)).float()


def _near(v, n, g):
    v = v.to(DEV)
    i = torch.randint(0, v.shape[0], (n,), generator=g, device=DEV)
    return v[i] + 0.02 * torch.randn((n, v.shape[1]), generator=g, device=DEV)


def _laid(x, soa):
    return x.t().contiguous() if soa else x.contiguous()


def _radii(n, g, lo, hi):
    return torch.rand(n, generator=g, device=DEV) * (hi - lo) + lo


def _split(n):
    n_cp, n_ray = n // 2, (3 * n) // 10
    return n_cp, n_ray, n - n_cp - n_ray


def _inputs(case, seed):
    """The inputs of a case as row-major tensors."""
    g, kind, n = _gen(seed), case["kind"], case.get("n")
    if kind == "cp3d":
        v, _ = _mesh_data(case["level"], AMPLITUDE[kind])
        return {"x": _near(v, n, g) if case["near"] else _box(n, 3, g)}
    if kind == "ray3d":
        return {"x": _box(n, 3, g), "v": _dirs(n, 3, g), "r": _radii(n, g, 0.1, 2.5) if case["r_max"] else None}
    if kind == "sil3d":
        return {"x": _box(n, 3, g), "r": _radii(n, g, 0.1, 1.5) if case["r_max"] else None}
    if kind == "cp2d":
        return {"x": _box(n, 2, g)}
    if kind == "wost2d":  # walkers between the inner (absorbing) and the outer (reflecting) boundary
        a = torch.rand(n, generator=g, device=DEV) * (2 * math.pi)
        r = torch.rand(n, generator=g, device=DEV) * 0.35 + 0.55
        return {"x": torch.stack([r * torch.cos(a), r * torch.sin(a)], 1), "v": _dirs(n, 2, g)}
    if kind == "batch2d":
        dim, geo = 2, [_line_data(m, seed=k)[0] for k, m in enumerate(_uneven(case["scenes"], case["segs"]))]
    else:
        dim = 3
        geo = [_mesh_data(3 + k % (case["level"] - 2), AMPLITUDE[kind], seed=k)[0] for k in range(case["scenes"])]
    weight = torch.tensor([float(v.shape[0]) for v in geo], device=DEV)
    mid = torch.stack([(v.amax(0) + v.amin(0)) / 2 for v in geo]).to(DEV)
    half = torch.stack([(v.amax(0) - v.amin(0)) / 2 for v in geo]).to(DEV)
    out = {}
    for name, k in zip(("cp", "ray", "sil"), _split(n)):
        ids = torch.multinomial(weight, k, replacement=True, generator=g).sort().values
        out[name] = (mid[ids] + half[ids] * _box(k, dim, g), ids.int())
    out["dir"] = _dirs(out["ray"][0].shape[0], dim, g)
    return out


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    if kind in ("cp3d", "ray3d", "sil3d"):
        s = {"kind": kind, "shape": _mesh(kind, case["level"])}
    elif kind == "cp2d":
        s = {"kind": kind, "shape": _line(case["segs"])}
    elif kind == "wost2d":
        s = {"kind": kind, "shape": _line(case["segs"]), "inner": _line(max(64, case["segs"] // 4), 0.4)}
    else:
        n_max = max(_split(case["n"]))
        if kind == "batch2d":
            b = SceneBatch(_batch2d(case["scenes"], case["segs"]), n_max)
        else:
            b = SceneBatch(_batch3d(case["scenes"], case["level"]), n_max, cp_variant="split", sil_variant="warp")
        s = {"kind": kind, "batch": b, "cp": (_laid(x["cp"][0], True), x["cp"][1]),
             "ray": (_laid(x["ray"][0], True), _laid(x["dir"], True), x["ray"][1]),
             "sil": (_laid(x["sil"][0], True), x["sil"][1])}
        return s
    s["x"] = _laid(x["x"], case["soa"])
    if "v" in x:
        s["v"] = _laid(x["v"], case["soa"])
    s["r"] = x.get("r")
    return s


def _fields(rec):
    return {k: v for k, v in vars(rec).items()}


def run(state):
    kind = state["kind"]
    if kind == "cp3d":
        return _fields(state["shape"].closest_point(state["x"]))
    if kind == "ray3d":
        r = math.inf if state["r"] is None else state["r"]
        return _fields(state["shape"].intersect(state["x"], state["v"], r))
    if kind == "sil3d":
        r = math.inf if state["r"] is None else state["r"]
        return _fields(state["shape"].closest_silhouette_snch(state["x"], r))
    if kind == "cp2d":
        return _fields(state["shape"].closest_point_bvh(state["x"]))
    if kind == "wost2d":
        cp = state["inner"].closest_point_bvh(state["x"])
        sil = state["shape"].closest_silhouette_snch(state["x"], cp.d)
        radius = torch.where(sil.valid, sil.d, cp.d)
        hit = state["shape"].intersect_bvh(state["x"], state["v"], radius)
        return {"cp": _fields(cp), "sil": _fields(sil), "hit": _fields(hit)}
    res = state["batch"].run(cp=state["cp"], ray=state["ray"], sil=state["sil"])
    return {"cp": _fields(res.cp), "ray": _fields(res.ray), "sil": _fields(res.sil)}


# ---- what a pass cannot do without ----------------------------------------------

def _geometry(kind, case):
    """(bytes of the vertices and indices, primitives) of the case's shapes."""
    if kind in ("cp3d", "ray3d", "sil3d"):
        f = [20 * 4 ** case["level"]]
        return sum(m // 2 * 12 + m * 12 for m in f), f[0]
    if kind == "cp2d":
        return case["segs"] * 16, case["segs"]
    if kind == "wost2d":
        return (case["segs"] + max(64, case["segs"] // 4)) * 16, case["segs"]
    if kind == "batch2d":
        m = _uneven(case["scenes"], case["segs"])
        return sum(m) * 16, max(m)
    f = [20 * 4 ** (3 + k % (case["level"] - 2)) for k in range(case["scenes"])]
    return sum(m // 2 * 12 + m * 12 for m in f), max(f)


def work(case):
    """Queries in, records out and the geometry once; a descent of a binary tree over the
    primitives (two box tests per level) and one primitive test per query."""
    kind, n = case["kind"], case["n"]
    geo, prims = _geometry(kind, case)
    depth = max(1.0, math.log2(prims))
    if kind == "cp3d":
        io, prim = 12 + 41, 100
    elif kind == "ray3d":
        io, prim = 24 + 42 + (4 if case["r_max"] else 0), 60
    elif kind == "sil3d":
        io, prim = 12 + 21 + (4 if case["r_max"] else 0), 80
    elif kind == "cp2d":
        io, prim = 8 + 29, 30
    elif kind == "wost2d":
        return {"bytes": float(geo + n * (8 + 29 + 8 + 4 + 17 + 16 + 4 + 30)), "flops": float(n * 3 * (depth * 24 + 30))}
    else:
        dim = 2 if kind == "batch2d" else 3
        n_cp, n_ray, n_sil = _split(n)
        per = ((8 + 4 + 29, 16 + 4 + 30, 8 + 4 + 17) if dim == 2 else (12 + 4 + 41, 24 + 4 + 42, 12 + 4 + 21))
        return {"bytes": float(geo + n_cp * per[0] + n_ray * per[1] + n_sil * per[2]),
                "flops": float(n * (depth * 12 * dim + 40 * dim - 50))}
    dim = 2 if kind == "cp2d" else 3
    return {"bytes": float(geo + n * io), "flops": float(n * (depth * 12 * dim + prim))}


# ---- the same in 64 bits ---------------------------------------------------------

def _tri_nearest(x, a, b, c):
    """Closest points of triangles (a, b, c) to x, broadcast, by the nearest of the three
    edges' segments and the projection onto the plane where it falls inside."""
    def dot(u, w):
        return (u * w).sum(-1, keepdim=True)

    def seg(p, q):
        u = q - p
        t = (dot(x - p, u) / dot(u, u)).clamp(0, 1)
        return p + t * u

    n = torch.cross(b - a, c - a, dim=-1)
    h = x - n * (dot(x - a, n) / dot(n, n))
    inside = ((dot(torch.cross(b - a, h - a, dim=-1), n) >= 0) & (dot(torch.cross(c - b, h - b, dim=-1), n) >= 0)
              & (dot(torch.cross(a - c, h - c, dim=-1), n) >= 0))
    best = torch.where(inside, h, torch.full_like(h, math.inf))
    d = torch.where(inside, (h - x).norm(dim=-1, keepdim=True), torch.full_like(inside, math.inf, dtype=x.dtype))
    for p, q in ((a, b), (b, c), (c, a)):
        s = seg(p, q)
        e = (s - x).norm(dim=-1, keepdim=True)
        best, d = torch.where(e < d, s, best), torch.minimum(d, e)
    return best, d.squeeze(-1)


def _cp_mesh64(x, v, f):
    """Closest points on a mesh: candidates are the triangles whose bounding sphere can hold
    a point nearer than the nearest vertex of the sphere-nearest triangle."""
    x, v, f = x.double(), v.to(DEV).double(), f.to(DEV).long()
    a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
    mid = (a + b + c) / 3
    rad = torch.stack([(q - mid).norm(dim=1) for q in (a, b, c)]).amax(0)
    p, d = torch.empty_like(x), torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 150_000_000 // f.shape[0])
    for k in range(0, x.shape[0], step):
        y = x[k:k + step]
        far = torch.cdist(y, mid)
        near = far.argmin(1)
        up = _tri_nearest(y, a[near], b[near], c[near])[1]
        i, j = torch.nonzero(far - rad <= up[:, None] + 1e-6, as_tuple=True)
        bd = torch.full((y.shape[0],), math.inf, device=DEV, dtype=torch.float64)
        qs, es = [], []
        for m in range(0, i.shape[0], 4_000_000):
            ii, jj = i[m:m + 4_000_000], j[m:m + 4_000_000]
            q, e = _tri_nearest(y[ii], a[jj], b[jj], c[jj])
            bd.scatter_reduce_(0, ii, e, "amin")
            qs.append(q)
            es.append(e)
        q, e = torch.cat(qs), torch.cat(es)
        won = e <= bd[i]
        p[k + i[won]] = q[won]
        d[k:k + step] = bd
    return p.t().contiguous(), d


def _cp_line64(x, v, e):
    x, v, e = x.double(), v.to(DEV).double(), e.to(DEV).long()
    a, u = v[e[:, 0]], v[e[:, 1]] - v[e[:, 0]]
    uu = (u * u).sum(1)
    p, d = torch.empty_like(x), torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 50_000_000 // e.shape[0])
    for k in range(0, x.shape[0], step):
        y = x[k:k + step]
        w0, w1 = y[:, :1] - a[:, 0], y[:, 1:] - a[:, 1]
        t = ((w0 * u[:, 0] + w1 * u[:, 1]) / uu).clamp(0, 1)
        q = (w0 - t * u[:, 0]).square() + (w1 - t * u[:, 1]).square()
        best, j = q.min(1)
        d[k:k + step] = best.sqrt()
        p[k:k + step] = a[j] + t.gather(1, j[:, None]) * u[j]
    return p.t().contiguous(), d


def _ray_mesh64(x, dirs, r, v, f):
    """(valid, point, distance) of the nearest hits, zeros on a miss."""
    x, dirs, v, f = x.double(), dirs.double(), v.to(DEV).double(), f.to(DEV).long()
    a, e1, e2 = v[f[:, 0]], v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]]
    t = torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 20_000_000 // f.shape[0])
    for k in range(0, x.shape[0], step):
        o, w = x[k:k + step, None], dirs[k:k + step, None]
        pv = torch.cross(w, e2[None], dim=-1)
        det = (e1 * pv).sum(-1)
        s = o - a
        u = (s * pv).sum(-1) / det
        q = torch.cross(s, e1[None].expand_as(s), dim=-1)
        m = (w * q).sum(-1) / det
        h = (e2 * q).sum(-1) / det
        ok = (u >= 0) & (m >= 0) & (u + m <= 1) & (h >= 0)
        t[k:k + step] = torch.where(ok, h, torch.full_like(h, math.inf)).amin(1)
    lim = math.inf if r is None else r.double()
    hit = (t <= lim) & (t < math.inf)
    t = torch.where(hit, t, torch.zeros_like(t))
    return hit, torch.where(hit[:, None], x + t[:, None] * dirs, torch.zeros_like(x)).t().contiguous(), t


def _ray_line64(x, dirs, v, e):
    x, dirs, v, e = x.double(), dirs.double(), v.to(DEV).double(), e.to(DEV).long()
    a, u = v[e[:, 0]], v[e[:, 1]] - v[e[:, 0]]
    t = torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 50_000_000 // e.shape[0])
    for k in range(0, x.shape[0], step):
        w0, w1 = x[k:k + step, :1] - a[:, 0], x[k:k + step, 1:] - a[:, 1]
        v0, v1 = dirs[k:k + step, :1], dirs[k:k + step, 1:]
        det = v0 * u[:, 1] - v1 * u[:, 0]
        s, h = (v0 * w1 - v1 * w0) / det, (u[:, 0] * w1 - u[:, 1] * w0) / det
        ok = (h > 0) & (s >= 0) & (s <= 1)
        t[k:k + step] = torch.where(ok, h, torch.full_like(h, math.inf)).amin(1)
    return torch.where(t < math.inf, t, torch.zeros_like(t))


def _edges(f):
    """Unique edges (a, b) of a closed mesh and the vertices opposite them in their two faces."""
    f = f.to(DEV).long()
    h = torch.cat([f[:, [0, 1, 2]], f[:, [1, 2, 0]], f[:, [2, 0, 1]]])
    key = torch.minimum(h[:, 0], h[:, 1]) * (1 << 32) + torch.maximum(h[:, 0], h[:, 1])
    h = h[key.argsort(stable=True)].reshape(-1, 2, 3)
    return h[:, 0, 0], h[:, 0, 1], h[:, 0, 2], h[:, 1, 2]


def _sil_mesh64(x, r, v, f):
    x, v = x.double(), v.to(DEV).double()
    a, b, c, e = (v[i] for i in _edges(f))
    u = b - a
    n0, n1, uu = torch.cross(u, c - a, dim=1), torch.cross(e - a, u, dim=1), (u * u).sum(1)
    d = torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 20_000_000 // a.shape[0])
    for k in range(0, x.shape[0], step):
        s = a - x[k:k + step, None]
        t = (-(s * u).sum(-1) / uu).clamp(0, 1)
        w = s + t[..., None] * u
        ok = ((w * n0).sum(-1) * (w * n1).sum(-1)) < 0
        d[k:k + step] = torch.where(ok, w.norm(dim=-1), torch.full_like(t, math.inf)).amin(1)
    lim = math.inf if r is None else r.double()
    return torch.where((d < lim) & (d < math.inf), d, torch.zeros_like(d))


def _sil_line64(x, r, v):
    """Silhouette vertices of a closed star polyline."""
    x, b = x.double(), v.to(DEV).double()
    a, c = b.roll(1, 0), b.roll(-1, 0)

    def side(p, q, y):
        return (q - p)[:, 0] * (y[:, 1:] - p[:, 1]) - (q - p)[:, 1] * (y[:, :1] - p[:, 0])

    d = torch.empty(x.shape[0], device=DEV, dtype=torch.float64)
    step = max(1, 50_000_000 // b.shape[0])
    for k in range(0, x.shape[0], step):
        y = x[k:k + step]
        ok = side(a, b, y) * side(b, c, y) < 0
        q = (y[:, :1] - b[:, 0]).square() + (y[:, 1:] - b[:, 1]).square()
        d[k:k + step] = torch.where(ok, q, torch.full_like(q, math.inf)).amin(1).sqrt()
    lim = math.inf if r is None else r.double()
    return torch.where((d < lim) & (d < math.inf), d, torch.zeros_like(d))


def _only(keys, **known):
    return {k: known.get(k) for k in keys}


CP3 = ("valid", "p", "n", "uv", "d", "prim_id")
CP2 = ("valid", "p", "n", "t", "d", "prim_id")
RAY3 = CP3 + ("on_boundary",)
RAY2 = CP2 + ("on_boundary",)
SIL = ("valid", "p", "d", "prim_id")


def exact(case, seed):
    """Distances and points in 64 bits (normals, coordinates and primitives of a point that
    several primitives share have no one value); None where it would take long."""
    kind = case["kind"]
    _, prims = _geometry(kind, case)
    pairs = case["n"] * prims
    if pairs > {"cp3d": 2e11, "ray3d": 2e9, "sil3d": 5e9, "cp2d": 2e10, "wost2d": 5e9, "batch2d": 7e10, "batch3d": 3e9}[kind]:
        return None
    x = _inputs(case, seed)
    if kind in ("cp3d", "ray3d", "sil3d"):
        v, f = _mesh_data(case["level"], AMPLITUDE[kind])
    if kind == "cp3d":
        p, d = _cp_mesh64(x["x"], v, f)
        return _only(CP3, p=p, d=d)
    if kind == "ray3d":
        _, p, d = _ray_mesh64(x["x"], x["v"], x["r"], v, f)
        return _only(RAY3, p=p, d=d)
    if kind == "sil3d":
        return _only(SIL, d=_sil_mesh64(x["x"], x["r"], v, f))
    if kind == "cp2d":
        p, d = _cp_line64(x["x"], *_line_data(case["segs"]))
        return _only(CP2, p=p, d=d)
    if kind == "wost2d":
        p, d = _cp_line64(x["x"], *_line_data(max(64, case["segs"] // 4), 0, 0.4))
        s = _sil_line64(x["x"], d, _line_data(case["segs"])[0])
        return {"cp": _only(CP2, p=p, d=d), "sil": _only(SIL, d=s), "hit": _only(RAY2)}
    out = {}
    for name in ("cp", "ray", "sil"):
        pts, ids = x[name]
        d = torch.zeros(pts.shape[0], device=DEV, dtype=torch.float64)
        p = torch.zeros((pts.shape[1], pts.shape[0]), device=DEV, dtype=torch.float64)
        for k in range(case["scenes"]):
            at = torch.nonzero(ids == k).flatten()
            if not at.numel():
                continue
            if kind == "batch2d":
                geo = _line_data(_uneven(case["scenes"], case["segs"])[k], seed=k)
            else:
                geo = _mesh_data(3 + k % (case["level"] - 2), AMPLITUDE[kind], seed=k)
            if name == "cp":
                p[:, at], d[at] = (_cp_line64 if kind == "batch2d" else _cp_mesh64)(pts[at], *geo)
            elif name == "ray":
                d[at] = (_ray_line64(pts[at], x["dir"][at], *geo) if kind == "batch2d" else
                         _ray_mesh64(pts[at], x["dir"][at], None, *geo)[2])
            else:
                d[at] = _sil_line64(pts[at], None, geo[0]) if kind == "batch2d" else _sil_mesh64(pts[at], None, *geo)
        keys = {"cp": CP2 if kind == "batch2d" else CP3, "ray": RAY2 if kind == "batch2d" else RAY3, "sil": SIL}[name]
        out[name] = _only(keys, p=p if name == "cp" else None, d=d)
    return out
