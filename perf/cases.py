"""Measured cases of the query paths: mesh signed distance (FP32, FP64, learned-seeded, DCEL and polygon
faces, moving geometry), nearest neighbours (tree and grid) and the CSG union, through the public
Python classes.

``listed()`` gives the fixed cases and ``draw(rng)`` further ones of the same ranges; ``prepare`` makes
the inputs and the handle that a program keeps, ``run`` is one pass, ``work`` what a pass cannot do
without, ``exact`` the 64-bit answer by exhaustive search in torch where that is affordable.
Meshes are displaced icospheres (20 * 4**level triangles) or displaced quad spheres (6 n^2 quads).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import ebgeometry_b200 as ebg
from ebgeometry_b200 import workloads as W

# candidate pairs (query, primitive) that exact() may look at
EXACT_PAIRS = 2.5e10


# --- the cases --------------------------------------------------------------------------------------

def listed():
    return [
        # one point at a time through ImplicitFunction::value: a program that walks a surface
        {"name": "value_one_l5", "kind": "value", "level": 5},
        # a few scattered points, as a particle or an interface step asks for
        {"name": "sdf_f32_l5_1k", "kind": "sdf", "level": 5, "points": "uniform", "n": 1000, "band": 0,
         "dtype": "float32", "seeded": False, "closest": False},
        # filling a level set on a Cartesian grid plus the cells near the surface, a 1.3 M-triangle mesh
        {"name": "sdf_f32_l8_grid512", "kind": "sdf", "level": 8, "points": "grid", "n": 512 ** 3, "band": 1 << 24,
         "dtype": "float32", "seeded": False, "closest": False},
        # the same level set through an attached learned model
        {"name": "sdf_f32_l8_grid512_seeded", "kind": "sdf", "level": 8, "points": "grid", "n": 512 ** 3,
         "band": 1 << 24, "dtype": "float32", "seeded": True, "closest": False},
        # FP64 in and out with the closest triangle: geometry set-up in double precision
        {"name": "sdf_f64_l5_1m", "kind": "sdf", "level": 5, "points": "uniform", "n": 1000000, "band": 0,
         "dtype": "float64", "seeded": False, "closest": True},
        # the DCEL-face distance of MeshSDF on an odd number of points
        {"name": "dcel_f64_l6_250k", "kind": "dcel", "level": 6, "n": 250007, "closest": False},
        # a quad mesh as a modelling program writes it
        {"name": "polygon_64_200k", "kind": "polygon", "side": 64, "mixed": False, "n": 200003},
        # the k nearest of a large clustered cloud
        {"name": "knn_16m_4m_k8", "kind": "knn", "cloud": 1 << 24, "clustered": True, "n": 1 << 22, "k": 8,
         "self": False},
        # a small lookup in a small cloud
        {"name": "knn_100k_1k_k1", "kind": "knn", "cloud": 100000, "clustered": True, "n": 1000, "k": 1, "self": False},
        # near-uniform particles on a hash grid
        {"name": "grid_4m_1m_k4", "kind": "grid_knn", "cloud": 1 << 22, "n": 1000003, "k": 4, "self": False},
        # a union of spheres and posed meshes evaluated on uneven batches
        {"name": "union_1024_48_2m", "kind": "union", "spheres": 1024, "meshes": 48, "n": 1 << 21, "batches": 61},
        # one step of moving geometry: new vertex positions, then a query
        {"name": "refit_l6_262k", "kind": "refit", "level": 6, "n": 262144},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choice(["value", "sdf", "sdf", "sdf", "sdf64", "dcel", "polygon", "knn", "knn", "grid_knn", "union",
                       "refit"])
    if kind == "value":
        return {"kind": kind, "level": rng.randint(3, 6)}
    if kind == "sdf":
        level = rng.randint(3, 8)
        points = rng.choice(["uniform", "grid", "band"])
        n = _log_int(rng, 1, 1 << 23)
        if points == "grid":
            n = max(2, round(n ** (1.0 / 3.0))) ** 3
        return {"kind": "sdf", "level": level, "points": points, "n": n, "band": n // 8 if points == "grid" else 0,
                "dtype": "float32", "seeded": level >= 5 and n >= 100000 and rng.random() < 0.5,
                "closest": rng.random() < 0.3}
    if kind == "sdf64":
        return {"kind": "sdf", "level": rng.randint(3, 6), "points": rng.choice(["uniform", "band"]),
                "n": _log_int(rng, 1, 1 << 20), "band": 0, "dtype": "float64", "seeded": False,
                "closest": rng.random() < 0.5}
    if kind == "dcel":
        return {"kind": kind, "level": rng.randint(3, 6), "n": _log_int(rng, 1, 1 << 19), "closest": rng.random() < 0.3}
    if kind == "polygon":
        return {"kind": kind, "side": _log_int(rng, 4, 96), "mixed": rng.random() < 0.5, "n": _log_int(rng, 1, 400000)}
    if kind == "knn":
        own = rng.random() < 0.3
        cloud = _log_int(rng, 1000, 1 << 21 if own else 1 << 24)
        return {"kind": kind, "cloud": cloud, "clustered": rng.random() < 0.7,
                "n": cloud if own else _log_int(rng, 1, 1 << 22), "k": _log_int(rng, 1, 32), "self": own}
    if kind == "grid_knn":
        own = rng.random() < 0.3
        cloud = _log_int(rng, 1000, 1 << 22)
        return {"kind": kind, "cloud": cloud, "n": cloud if own else _log_int(rng, 1, 1 << 20),
                "k": _log_int(rng, 1, 16), "self": own}
    if kind == "union":
        return {"kind": kind, "spheres": _log_int(rng, 1, 2048), "meshes": rng.randint(0, 48),
                "n": _log_int(rng, 1, 1 << 22), "batches": rng.randint(1, 64)}
    return {"kind": "refit", "level": rng.randint(3, 7), "n": _log_int(rng, 1, 1 << 20)}


# --- inputs -----------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return W.icosphere(level)


@functools.lru_cache(maxsize=None)
def _quad_sphere(side, mixed):
    """Unit directions and (offsets, indices) of the quad sphere; its faces do not depend on the seed."""
    v, f = (W.mixed_polygon_sphere if mixed else W.displaced_quad_sphere)(side, 0)
    return v / np.linalg.norm(v, axis=1, keepdims=True), f


def _displaced(u, seed, radius=1.0):
    a, w, phi = W.radial_field(seed)
    return (radius * (1.0 + (np.sin(u @ w.T + phi) * a).sum(axis=1)))[:, None] * u


def _mesh(level, seed, radius=1.0):
    u, f = _icosphere(level)
    return _displaced(u, seed, radius), f


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, seed, dtype=torch.float32, lo=-1.5, hi=1.5):
    return torch.rand((n, 3), generator=_generator(seed), device="cuda", dtype=dtype) * (hi - lo) + lo


def _grid(n, lo=-1.25, hi=1.25):
    res = round(n ** (1.0 / 3.0))
    c = (lo + (hi - lo) / res * (torch.arange(res, device="cuda", dtype=torch.float64) + 0.5)).float()
    out = torch.empty((res, res, res, 3), device="cuda")
    out[..., 0] = c[None, None, :]
    out[..., 1] = c[None, :, None]
    out[..., 2] = c[:, None, None]
    return out.reshape(-1, 3)


def _near(v, f, n, seed, width=1e-3):
    """Points within +-width of the surface, triangles drawn by area."""
    g = _generator(seed)
    x = torch.from_numpy(v).cuda()[torch.from_numpy(f.astype(np.int64)).cuda()]
    cr = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
    area = cr.norm(dim=1)
    cdf = torch.cumsum(area, 0)
    pick = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
    tri = torch.searchsorted(cdf, pick).clamp_(max=f.shape[0] - 1)
    r = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    s = r[:, 0].sqrt()
    p = (1.0 - s)[:, None] * x[tri, 0]
    p += (s * (1.0 - r[:, 1]))[:, None] * x[tri, 1]
    p += (s * r[:, 1])[:, None] * x[tri, 2]
    p += ((2.0 * r[:, 2] - 1.0) * width)[:, None] * (cr / area[:, None])[tri]
    return p


def _queries(case, v, f, seed):
    dtype = torch.float64 if case.get("dtype", "float32") == "float64" else torch.float32
    if case["points"] == "uniform":
        return _uniform(case["n"], seed, dtype)
    if case["points"] == "band":
        return _near(v, f, case["n"], seed).to(dtype).contiguous()
    p = _grid(case["n"])
    return torch.cat([p, _near(v, f, case["band"], seed).float()]) if case["band"] else p


def _cloud(n, seed, clustered):
    """Uniform in the unit cube; clustered: half of it from 64 anisotropic Gaussian clusters."""
    g = _generator(seed)
    nu = n // 2 if clustered else n
    out = torch.empty((n, 3), device="cuda")
    out[:nu] = torch.rand((nu, 3), generator=g, device="cuda")
    if n > nu:
        m = n - nu
        lab = torch.randint(64, (m,), generator=g, device="cuda")
        cen = torch.rand((64, 3), generator=g, device="cuda")
        lo, hi = math.log(0.002), math.log(0.05)
        sig = torch.exp(torch.rand((64, 3), generator=g, device="cuda") * (hi - lo) + lo)
        rot = torch.linalg.qr(torch.randn((64, 3, 3), generator=g, device="cuda", dtype=torch.float64))[0].float()
        z = torch.randn((m, 3), generator=g, device="cuda") * sig[lab]
        basis = rot[lab]
        out[nu:] = ((basis * z[:, None, :]).sum(-1) + cen[lab]).clamp_(0.0, 1.0)
    return out


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    s, m = case["spheres"], case["meshes"]
    spheres = np.concatenate([rng.uniform(-1, 1, (s, 3)),
                              np.exp(rng.uniform(math.log(0.001), math.log(0.05), (s, 1)))], axis=1)
    meshes, poses = [], np.empty((m, 5))
    for i in range(m):
        meshes.append((*_mesh(3 + i % 3, int(rng.integers(1 << 30)), float(rng.uniform(0.03, 0.12))),))
        poses[i] = [rng.uniform(0, 360), rng.integers(0, 3), *rng.uniform(-1, 1, 3)]
    return spheres, meshes, poses


def _batch_sizes(case):
    """Uneven batch sizes that add up to n, none empty while there are points for all."""
    b = min(case["batches"], case["n"])
    w = np.random.default_rng(case["n"]).uniform(0.2, 1.8, b)
    cut = np.round(np.cumsum(w) / w.sum() * (case["n"] - b)).astype(np.int64)
    return [int(x) + 1 for x in np.diff(np.concatenate([[0], cut]))]


def _inputs(case, seed):
    """The raw inputs, shared by prepare() and exact()."""
    kind = case["kind"]
    if kind == "value":
        v, f = _mesh(case["level"], seed)
        return v, f, np.random.default_rng(seed).uniform(-1.5, 1.5, 3)
    if kind in ("sdf", "dcel"):
        v, f = _mesh(case["level"], seed)
        c = case if kind == "sdf" else dict(case, points="uniform", dtype="float64")
        return v, f, _queries(c, v, f, seed)
    if kind == "polygon":
        u, f = _quad_sphere(case["side"], case["mixed"])
        return _displaced(u, seed), f, _uniform(case["n"], seed, torch.float64)
    if kind in ("knn", "grid_knn"):
        pts = _cloud(case["cloud"], seed, case.get("clustered", False))
        return pts, None if case["self"] else torch.rand((case["n"], 3), generator=_generator(seed + 1), device="cuda")
    if kind == "union":
        pts = _uniform(case["n"], seed, lo=-1.2, hi=1.2)
        return (*_scene(case, seed), [p.contiguous() for p in pts.split(_batch_sizes(case))])
    v, f = _mesh(case["level"], seed)
    moved = _displaced(_icosphere(case["level"])[0], seed + 1)
    return v, f, moved, _uniform(case["n"], seed)


def prepare(case, seed):
    kind = case["kind"]
    made = _inputs(case, seed)
    state = {"kind": kind, "case": case}
    if kind in ("value", "sdf", "dcel", "refit"):
        cls = ebg.MeshSDF if kind == "dcel" else ebg.TriMeshSDF
        large = case["level"] >= 7
        state["mesh"] = cls(made[0], made[1], build="Morton" if large else "SAH", on_device=large)
    if kind == "value":
        state["point"] = tuple(float(x) for x in made[2])
    elif kind == "sdf":
        state["points"] = made[2]
        state["seed"] = None
        if case["seeded"]:
            state["seed"] = ebg.SeedModel.train(state["mesh"], num_samples=1 << 21, steps=300, batch=1 << 16, rng_seed=1,
                                                lo=[-1.25] * 3, hi=[1.25] * 3)
        state["closest"] = torch.empty(made[2].shape[0], dtype=torch.int32, device="cuda") if case["closest"] else None
    elif kind == "dcel":
        state["points"] = made[2]
        state["closest"] = torch.empty(made[2].shape[0], dtype=torch.int32, device="cuda") if case["closest"] else None
    elif kind == "polygon":
        state["mesh"] = ebg.PolygonMeshSDF(made[0], made[1])
        state["points"] = made[2]
    elif kind == "knn":
        state["cloud"], state["queries"] = ebg.PointCloudBVH(made[0]), made[1]
    elif kind == "grid_knn":
        state["cloud"], state["queries"] = ebg.PointCloudHashGrid(made[0].cpu().numpy()), made[1]
    elif kind == "union":
        meshes = [ebg.TriMeshSDF(v, f, build="Morton", on_device=True) for v, f in made[1]]
        state["scene"], state["batches"] = ebg.BVHUnion(made[0], meshes, made[2]), made[3]
    elif kind == "refit":
        state["vertices"], state["points"] = torch.from_numpy(made[2]).cuda(), made[3]
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "value":
        return state["mesh"].value(state["point"])
    if kind == "sdf":
        return state["mesh"].signed_distance(state["points"], closest_tri=state["closest"], seed=state["seed"])
    if kind == "dcel":
        return state["mesh"].signed_distance(state["points"], closest_tri=state["closest"])
    if kind == "polygon":
        return state["mesh"].signed_distance(state["points"])
    if kind in ("knn", "grid_knn"):
        if state["queries"] is None:
            return state["cloud"].all_nearest_neighbors(case["k"], device=True)
        return state["cloud"].knn(state["queries"], case["k"])
    if kind == "union":
        return state["scene"].values_batches(state["batches"])
    state["mesh"].refit(state["vertices"])
    return state["mesh"].signed_distance(state["points"])


# --- what a pass cannot do without ------------------------------------------------------------------

def work(case):
    """Bytes: geometry, queries and results once each.  Operations: a descent of a 4-wide tree (four
    box distances of 11 operations a level) and one leaf (8 triangles of about 60 operations, or 8
    points of 8) a query."""
    kind = case["kind"]

    def search(n, prims, leaf_ops):
        levels = max(1.0, math.log(max(2.0, prims / 8.0), 4.0))
        return n * (44.0 * levels + leaf_ops)

    if kind in ("knn", "grid_knn"):
        n, k = case["n"], case["k"]
        q = 0 if case["self"] else 12 * n
        return {"bytes": 12.0 * case["cloud"] + q + 8.0 * n * k, "flops": search(n, case["cloud"], 64.0)}
    if kind == "union":
        tris = sum(20 * 4 ** (3 + i % 3) for i in range(case["meshes"]))
        return {"bytes": 16.0 * case["spheres"] + 36.0 * tris + 16.0 * case["n"],
                "flops": search(case["n"], tris + case["spheres"], 480.0)}
    if kind == "polygon":
        faces = 6 * case["side"] ** 2
        return {"bytes": 96.0 * faces + 32.0 * case["n"], "flops": search(case["n"], faces, 640.0)}
    tris = 20 * 4 ** case["level"]
    n = case.get("n", 1) + case.get("band", 0)
    wide = kind in ("value", "dcel") or case.get("dtype") == "float64"
    per = (32 if wide else 16) + (4 if case.get("closest") else 0)
    moved = 12.0 * tris + 12.0 * tris if kind == "refit" else 0.0
    return {"bytes": (72.0 if wide else 36.0) * tris + moved + float(per) * n, "flops": search(n, tris, 480.0)}


# --- the answers in 64 bits ---------------------------------------------------------------------------

def _padded_faces(v, faces):
    """(F, K, 3) corners and (F,) corner counts of triangles (T, 3) or (offsets, indices) faces."""
    x = torch.from_numpy(np.ascontiguousarray(v, np.float64)).cuda()
    if isinstance(faces, tuple):
        off, idx = faces
        count = np.diff(off)
        at = off[:-1, None] + np.minimum(np.arange(count.max()), count[:, None] - 1)
        tab = idx[at]
    else:
        tab, count = faces, np.full(faces.shape[0], 3)
    return x[torch.from_numpy(np.ascontiguousarray(tab, np.int64)).cuda()], torch.from_numpy(count).cuda()


def _face_distance(p, x, cnt, nrm, cen):
    """Unsigned distance of points (M, 3) to faces (M, K, 3): |n . (p - c)| where the projection into
    the face's plane lies inside it (crossing number, largest normal axis dropped), else the nearest
    edge point."""
    drop = nrm.abs().argmax(dim=1)
    ax = torch.where(drop == 0, 1, 0)[:, None]
    ay = torch.where(drop == 2, 1, 2)[:, None]
    h = (nrm * (p - cen)).sum(1)
    q = p - h[:, None] * nrm
    qx, qy = q.gather(1, ax)[:, 0], q.gather(1, ay)[:, 0]
    crossings = torch.zeros_like(drop)
    best = torch.full_like(h, math.inf)
    k = x.shape[1]
    for i in range(k):
        a = x[:, i]
        last = cnt <= i + 1
        b = torch.where(last[:, None], x[:, 0], x[:, (i + 1) % k])
        used = cnt > i
        a2x, a2y, b2x, b2y = a.gather(1, ax)[:, 0], a.gather(1, ay)[:, 0], b.gather(1, ax)[:, 0], b.gather(1, ay)[:, 0]
        span = ((a2y <= qy) & (b2y > qy)) | ((a2y > qy) & (b2y <= qy))
        t = (qy - a2y) / torch.where(span, b2y - a2y, 1.0)
        crossings += (used & span & (qx < a2x + t * (b2x - a2x))).long()
        e = b - a
        s = ((p - a) * e).sum(1) / torch.where(used, (e * e).sum(1), 1.0)
        d = (p - a - s.clamp(0.0, 1.0)[:, None] * e).norm(dim=1)
        best = torch.where(used & (d < best), d, best)
    return torch.where(crossings % 2 == 1, h.abs(), best)


def _surface_distance(v, faces, pts):
    """Signed distance of FP64 CUDA points to a mesh that is star-shaped about the origin, or None
    where that is too much work."""
    x, cnt = _padded_faces(v, faces)
    if x.shape[0] * pts.shape[0] > EXACT_PAIRS:
        return None
    cr = torch.linalg.cross(x[:, 2] - x[:, 0], x[:, 2] - x[:, 1])
    nrm = cr / cr.norm(dim=1, keepdim=True)
    live = (torch.arange(x.shape[1], device="cuda")[None] < cnt[:, None])
    cen = (x * live[..., None]).sum(1) / cnt[:, None]
    rad = (x - cen[:, None]).norm(dim=2).amax(1)
    # the cone of each face over the origin, in triangles: three inward planes each
    tri = [x[:, [0, i, i + 1]] for i in range(1, x.shape[1] - 1)]
    cone = torch.cat([t[live[:, i + 2]] for i, t in enumerate(tri)])
    side = [torch.linalg.cross(cone[:, i], cone[:, (i + 1) % 3]) for i in range(3)]
    side = [s / s.norm(dim=1, keepdim=True) for s in side]
    face = torch.linalg.cross(cone[:, 1] - cone[:, 0], cone[:, 2] - cone[:, 0])
    off = (face * cone[:, 0]).sum(1)
    out = torch.empty(pts.shape[0], dtype=torch.float64, device="cuda")
    step = max(1, int(1.5e8) // x.shape[0])
    c2 = (cen * cen).sum(1)
    for b in range(0, pts.shape[0], step):
        p = pts[b:b + step]
        d = ((p * p).sum(1)[:, None] + c2[None] - 2.0 * (p @ cen.T)).clamp_(min=0.0).sqrt_()
        upper = (d + rad[None]).amin(1) * (1.0 + 1e-6) + 1e-6
        i, j = torch.nonzero(d - rad[None] * 1.02 - 1e-6 <= upper[:, None], as_tuple=True)
        del d
        near = torch.full((p.shape[0],), math.inf, dtype=torch.float64, device="cuda")
        for s in range(0, i.numel(), 1 << 24):
            ii, jj = i[s:s + (1 << 24)], j[s:s + (1 << 24)]
            near.scatter_reduce_(0, ii, _face_distance(p[ii], x[jj], cnt[jj], nrm[jj], cen[jj]), "amin")
        w = p @ side[0].T
        for q in side[1:]:
            torch.minimum(w, p @ q.T, out=w)
        t = w.argmax(1)
        del w
        sign = torch.where((face[t] * p).sum(1) < off[t], -1.0, 1.0)
        out[b:b + step] = sign * near
    return out


def _rotated(p, angle, axis):
    c, s = math.cos(angle * math.pi / 180.0), math.sin(angle * math.pi / 180.0)
    x, y, z = p.unbind(1)
    if axis == 0:
        return torch.stack([x, y * c + z * s, -y * s + z * c], 1)
    if axis == 1:
        return torch.stack([x * c - z * s, y, x * s + z * c], 1)
    return torch.stack([x * c + y * s, -x * s + y * c, z], 1)


def _union(made):
    spheres, meshes, poses, batches = made
    p = torch.cat(batches).double()
    best = torch.full((p.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    for s in torch.from_numpy(spheres).cuda():
        torch.minimum(best, (p - s[:3]).norm(dim=1) - s[3], out=best)
    local, reach = [], best.clone()
    for (v, _), pose in zip(meshes, poses):
        r = np.linalg.norm(v, axis=1)
        dist = (p - torch.from_numpy(pose[2:]).cuda()).norm(dim=1)
        local.append((dist, r.max()))
        torch.minimum(reach, (dist - 0.97 * r.min()).clamp(min=0.0), out=reach)
    pairs = sum(int((d - r <= reach).sum()) * f.shape[0] for (d, r), (_, f) in zip(local, meshes))
    if pairs > EXACT_PAIRS:
        return None
    for (dist, r), (v, f), pose in zip(local, meshes, poses):
        near = torch.nonzero(dist - r <= reach)[:, 0]
        if near.numel():
            q = _rotated(p[near] - torch.from_numpy(pose[2:]).cuda(), pose[0], int(pose[1]))
            best[near] = torch.minimum(best[near], _surface_distance(v, f, q))
    return [x.cpu() for x in best.split([b.shape[0] for b in batches])]


def _nearest(case, pts, queries):
    """Squared distances of the k nearest (FP32 coordinates, FP64 arithmetic)."""
    p = pts.double()
    q = p if queries is None else queries.double()
    if float(p.shape[0]) * q.shape[0] > EXACT_PAIRS / 4:
        return None
    out = torch.empty((q.shape[0], case["k"]), dtype=torch.float64, device="cuda")
    step = max(1, int(1e8) // p.shape[0])
    for b in range(0, q.shape[0], step):
        x = q[b:b + step]
        d = (x[:, None, 0] - p[None, :, 0]).square_()
        for a in (1, 2):
            d += (x[:, None, a] - p[None, :, a]).square_()
        if queries is None:
            d[torch.arange(x.shape[0]), torch.arange(b, b + x.shape[0])] = math.inf
        out[b:b + step] = d.topk(case["k"], dim=1, largest=False, sorted=True)[0]
    return out.cpu()


def exact(case, seed):
    kind = case["kind"]
    made = _inputs(case, seed)
    if kind == "value":
        return float(_surface_distance(made[0], made[1], torch.from_numpy(made[2][None]).cuda())[0])
    if kind in ("sdf", "dcel"):
        n = made[2].shape[0]
        d = _surface_distance(made[0], made[1], made[2].double()) if n * made[1].shape[0] <= EXACT_PAIRS else None
        d = None if d is None else d.cpu()
        return (d, None) if case["closest"] and d is not None else d
    if kind == "polygon":
        d = _surface_distance(made[0], made[1], made[2])
        return None if d is None else d.cpu()
    if kind in ("knn", "grid_knn"):
        d = _nearest(case, made[0], made[1])
        return None if d is None else (None, d)
    if kind == "union":
        return _union(made)
    d = _surface_distance(made[2], made[1], made[3].double())
    return None if d is None else d.cpu()
