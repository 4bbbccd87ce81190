"""The calls a program makes of this library, as measurable cases.

Each case is one pass through a public entry point (beamtrace2007_b200.renderer,
beamtrace2007_b200.serving) with host or device buffers as that entry point takes
them.  A seed moves the camera and the light (or the meshes): the scene files a
program loads stay the same from frame to frame, what it looks at does not.

Kinds
    soft    GpuRenderer.soft_shadows: a frame of area-light shadows, images to the host
    points  GpuRenderer.soft_points: supplied shading points (lightmap texels), host arrays
    ids     GpuRenderer.primary_ids: per-pixel visible triangle ids
    mask    GpuRenderer.point_mask: ids and the shadow mask of a point light
    polys   GpuRenderer.primary, point_shadows, raster: exact polygons to the host and back
    batch   GpuRenderer.batch_soft: several jobs over a pool of scenes, outputs on the device
    kd      PreparedScene with the kd-tree built on the GPU: what a program pays per new mesh
    serve   serving.Server: a burst of mixed requests over two resident scenes
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from beamtrace2007_b200 import scenes
from beamtrace2007_b200.renderer import GpuRenderer, PreparedScene, make_camera


def listed():
    return [
        # a preview thumbnail: latency and launches
        {"name": "soft_room_64x48", "kind": "soft", "scene": "room", "W": 64, "H": 48, "scale": 1.0, "exact": True},
        # the headline frame of the benchmark
        {"name": "soft_plant_512", "kind": "soft", "scene": "plant", "W": 512, "H": 512, "scale": 1.0, "exact": True},
        # an odd-sized viewport under a wide light, Lambert factor at the light's centre
        {"name": "soft_plant_333x217_wide", "kind": "soft", "scene": "plant", "W": 333, "H": 217, "scale": 4.0,
         "exact": False},
        # a dense mesh that does not sit in L1: the largest case
        {"name": "soft_sphere_512", "kind": "soft", "scene": "sphere7", "W": 512, "H": 512, "scale": 2.0,
         "exact": True},
        # lightmap texels baked through supplied points
        {"name": "points_plant_4801", "kind": "points", "scene": "plant", "n": 4801, "scale": 0.5, "exact": True},
        # picking in a simple scene at the reference's tile
        {"name": "ids_room_256", "kind": "ids", "scene": "room", "W": 256, "H": 256, "tile": 16},
        # a visibility buffer of a detailed interior at the serving tile
        {"name": "ids_meeting_1024", "kind": "ids", "scene": "meeting", "W": 1024, "H": 1024, "tile": 4},
        # a point light's shadow mask in a large building
        {"name": "mask_building_1024", "kind": "mask", "scene": "building2", "W": 1024, "H": 1024, "tile": 16},
        # the polygon interface of the reference's GpuRenderer, at its tile
        {"name": "polys_building_511x389", "kind": "polys", "scene": "building2", "W": 511, "H": 389, "tile": 16},
        # a queue of small jobs over many scenes
        {"name": "batch_12_jobs", "kind": "batch", "jobs": 12, "tris": 20000, "size": 128},
        # a mesh a program has just loaded
        {"name": "kd_sphere7", "kind": "kd", "scene": "sphere7"},
        # a burst of requests of every kind at a server
        {"name": "serve_mixed_12", "kind": "serve", "requests": 12, "size": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["soft", "soft", "soft", "soft", "points", "ids", "mask", "polys", "batch", "kd", "serve"])
    if kind == "soft":
        scene = rng.choice(["room", "plant", "plant", "sphere4", "sphere5", "sphere7", "meeting"])
        big = {"room": 700, "plant": 512, "meeting": 300}.get(scene, 512)
        wide = {"room": 4.0, "plant": 2.0, "meeting": 1.0}.get(scene, 1.5)
        W, H = _log_int(rng, 17, big), _log_int(rng, 17, big)
        if scene == "plant" and W * H < 100000:
            wide = 4.0
        return {"kind": kind, "scene": scene, "W": W, "H": H,
                "scale": round(math.exp(rng.uniform(math.log(0.25), math.log(wide))), 3),
                "exact": rng.random() < 0.6}
    if kind == "points":
        return {"kind": kind, "scene": rng.choice(["room", "plant", "sphere5"]), "n": _log_int(rng, 1, 60000),
                "scale": round(rng.uniform(0.25, 1.5), 3), "exact": rng.random() < 0.6}
    if kind in ("ids", "mask", "polys"):
        # (point shadows of a curved mesh's sliver hits can need a clip the library refuses:
        # a few camera positions in a hundred)
        scene = rng.choice(["room", "plant", "sphere4", "sphere5", "meeting", "building2"] if kind == "ids" else
                           ["room", "building2"])
        W, H = _log_int(rng, 33, 1024), _log_int(rng, 33, 1024)
        tile = rng.choice([2, 4, 8, 16] if kind == "polys" else [1, 2, 3, 4, 8, 16])
        while (W // tile) * (H // tile) > 1 << 18:
            tile *= 2
        if scene == "meeting":  # larger tiles over a dense mesh: the library's tuner does not pick them
            tile, W, H = min(tile, 4), max(W, 256), max(H, 200)
        return {"kind": kind, "scene": scene, "W": W, "H": H, "tile": tile}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randrange(2, 16), "tris": _log_int(rng, 500, 20000),
                "size": rng.randrange(33, 129)}
    if kind == "kd":
        return {"kind": kind, "scene": rng.choice(["room", "plant", "sphere3", "sphere4", "sphere5", "sphere6",
                                                   "meeting"])}
    return {"kind": kind, "requests": rng.randrange(3, 15), "size": rng.randrange(65, 257)}


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _scene(name):
    if name.startswith("sphere"):
        return scenes.displaced_sphere(int(name[6:]))
    if name == "building2":
        return scenes.building(floors=2)
    return scenes.SCENES[name]()


@functools.lru_cache(maxsize=None)
def _prepared(name):
    s = _scene(name)
    return PreparedScene(s.pos, s.tris, kd_device=0)


@functools.lru_cache(maxsize=None)
def _job(seed, tris):
    s = scenes.shadow_job(seed, tris)
    return s, PreparedScene(s.pos, s.tris, kd_device=0)


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, len(case["kind"])])


def _view(s, rng):
    """The scene's view with the eye moved a little (relative to its distance to the target)."""
    v = s.views[0]
    e, t = np.asarray(v.eye, np.float64), np.asarray(v.target, np.float64)
    e = e + rng.uniform(-0.02, 0.02, 3) * np.linalg.norm(t - e)
    return e.astype(np.float32), t.astype(np.float32), float(v.fov)


def _area_light(s, rng, scale):
    L = s.light_array(scale)
    L[:3] += rng.uniform(-0.04, 0.04, 3)
    return L.astype(np.float32).astype(np.float64)


def _point_light(s, rng):
    return (np.asarray(s.point_light, np.float64) + rng.uniform(-0.04, 0.04, 3)).astype(np.float32)


def _surface_points(s, rng, n):
    """Points spread over the scene's surfaces by area, with the side that faces the light."""
    P = s.pos[s.tris.astype(np.int64)].astype(np.float64)
    nrm = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    area = np.linalg.norm(nrm, axis=1)
    tri = rng.choice(len(P), size=n, p=area / area.sum())
    u, v = rng.uniform(0.02, 0.98, n), rng.uniform(0.02, 0.98, n)
    flip = u + v > 1
    u, v = np.where(flip, 1 - u, u), np.where(flip, 1 - v, v)
    X = P[tri, 0] + u[:, None] * (P[tri, 1] - P[tri, 0]) + v[:, None] * (P[tri, 2] - P[tri, 0])
    N = nrm[tri] / area[tri, None]
    N *= np.where(np.einsum("ij,ij->i", N, np.asarray(s.area_light[0]) - X) < 0, -1.0, 1.0)[:, None]
    return tri.astype(np.int32), X.astype(np.float32), N.astype(np.float32)


def _inputs(case, seed):
    """What the seed decides, as host arrays (shared by prepare and exact)."""
    rng = _rng(case, seed)
    k = case["kind"]
    if k in ("soft", "points"):
        s = _scene(case["scene"])
        d = {"light": _area_light(s, rng, case["scale"])}
        if k == "soft":
            d["view"] = _view(s, rng)
        else:
            d["tri"], d["X"], d["N"] = _surface_points(s, rng, case["n"])
        return d
    if k in ("ids", "mask", "polys"):
        s = _scene(case["scene"])
        return {"view": _view(s, rng), "light": _point_light(s, rng)}
    if k == "kd":
        s = _scene(case["scene"])
        # the same mesh exported with its triangles in another order
        return {"pos": s.pos, "tris": np.ascontiguousarray(s.tris[rng.permutation(len(s.tris))])}
    if k == "batch":
        jobs = []
        for j in range(case["jobs"]):
            tris = max(200, int(case["tris"] * (j + 1) / case["jobs"]))
            s = _job(100 + j, tris)[0]
            size = case["size"] if j % 2 == 0 else max(33, case["size"] // 2 + 3)
            jobs.append((j, tris, size, _view(s, rng), _area_light(s, rng, float(rng.uniform(0.25, 2.0)))))
        return {"jobs": jobs}
    kinds = ["primary", "soft", "point"]
    reqs = [(kinds[j % 3], ("plant", "sphere5")[(j // 2) % 2],
             case["size"] if j % 2 == 0 else case["size"] // 2 + 1, float(rng.choice([0.5, 1.0, 1.5])))
            for j in range(case["requests"])]
    moved = []
    for name in ("plant", "sphere5"):
        s = _scene(name)
        moved.append((name, _view(s, rng), _area_light(s, rng, 1.0), _point_light(s, rng)))
    return {"requests": reqs, "scenes": moved}


def _camera(s, view, W, H):
    return make_camera(view[0], view[1], view[2], s.up, W, H)


class _Burst:
    """A running server, closed with the state."""

    def __init__(self, moved):
        import copy

        from beamtrace2007_b200.serving import Server
        self.server = Server({name: _prepared(name) for name, *_ in moved}, queue_records=1 << 22)
        for name, view, light, point in moved:
            s = copy.copy(_scene(name))
            s.views = [scenes.View(tuple(view[0]), tuple(view[1]), view[2])]
            s.area_light = (light[:3], light[3:6], light[6:])
            s.point_light = tuple(float(x) for x in point)
            self.server.scenes[name].data = s

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    k, d = case["kind"], _inputs(case, seed)
    d["kind"] = k
    if k == "kd":
        return d
    if k == "serve":
        d["burst"] = _Burst(d["scenes"])
        return d
    if k == "batch":
        first = _job(100, d["jobs"][0][1])[1]
        g = GpuRenderer(first)
        d["ids"] = [0] + [g.add_scene(_job(100 + j, tris)[1]) for j, tris, *_ in d["jobs"][1:]]
        d["cams"] = [_camera(_job(100 + j, tris)[0], view, size, size) for j, tris, size, view, _ in d["jobs"]]
        d["lights"] = [x[4] for x in d["jobs"]]
    else:
        g = GpuRenderer(_prepared(case["scene"]))
        if k != "points":
            d["cam"] = _camera(_scene(case["scene"]), d["view"], case["W"], case["H"])
    d["g"] = g
    d["case"] = case
    return d


def run(state):
    k, g = state["kind"], state.get("g")
    if k == "kd":
        ps = PreparedScene(state["pos"], state["tris"], kd_device=0)
        return {n: getattr(ps, n) for n in ("tris", "tri_normals", "tri_area", "bounds", "kd_split", "kd_data",
                                            "kd_offset", "kd_parent", "kd_box", "kd_tri_indices", "kd_bounds")}
    if k == "serve":
        from beamtrace2007_b200.serving import Request
        srv = state["burst"].server
        rs = [srv.submit(Request(kind, name, size, size, light_scale=scale))
              for kind, name, size, scale in state["requests"]]
        for r in rs:
            r.event.wait()
        if any(r.error for r in rs):
            raise RuntimeError(next(r.error for r in rs if r.error))
        return [{"tri": r.result.tri, "vis": r.result.vis, "E": r.result.E, "Eu": r.result.Eu} if r.kind == "soft"
                else r.result for r in rs]
    case = state["case"]
    if k == "soft":
        r = g.soft_shadows(state["cam"], state["light"], exact=case["exact"])
        return {"tri": r.tri, "vis": r.vis, "E": r.E, "Eu": r.Eu}
    if k == "points":
        r = g.soft_points(state["light"], state["tri"], state["X"], state["N"], exact=case["exact"])
        return {"vis": r.vis, "E": r.E, "Eu": r.Eu}
    if k == "ids":
        return g.primary_ids(state["cam"], tile=case["tile"])
    if k == "mask":
        ids, mask = g.point_mask(state["cam"], state["light"], tile=case["tile"])
        return {"ids": ids, "mask": mask}
    if k == "polys":
        prim = g.primary(state["cam"], tile=case["tile"])
        sh = g.point_shadows(state["cam"], prim, state["light"])
        # the polygons come in no fixed order: the images made of them stand for them
        ids, mask = g.raster(state["cam"], prim, sh)
        return {"ids": ids, "mask": mask}
    outs, _ = g.batch_soft(state["cams"], state["lights"], exact=True, device_outputs=True, scenes=state["ids"])
    return [{"tri": t, "vis": v, "E": e, "Eu": u} for t, v, e, u in outs]


# -------------------------------------------------------------------- work

# Beam-triangle tests a shadow root needs at light scale 1 (the tracer's counters, which
# the algorithm fixes), and the power of the scale they grow with.
_TESTS = {"room": (34, 1.0), "plant": (77, 1.8), "meeting": (250, 1.0), "sphere": (100, 1.4), "job": (2000, 1.6)}
# Tests per pixel of primary tiles and of primary tiles with point shadows.
_TILE_TESTS = {"room": 0.5, "plant": 8, "meeting": 18, "sphere4": 8, "sphere5": 15, "building2": 0.4}
_FLOPS = 160  # one test: three edge planes and lines, 12 corner votes, its share of the tree walk


def _family(name):
    return "sphere" if name.startswith("sphere") else name


def _scene_bytes(name):
    """Positions, indices, and a kd-tree of about 1.5 nodes (8 bytes) and 2 references (4 bytes) per triangle."""
    s = _scene(name)
    return s.pos.nbytes + s.tris.nbytes + 20 * len(s.tris)


def work(case):
    k = case["kind"]
    if k in ("soft", "points"):
        n = case["W"] * case["H"] if k == "soft" else case["n"]
        t, p = _TESTS[_family(case["scene"])]
        return {"bytes": _scene_bytes(case["scene"]) + n * (16 if k == "soft" else 28 + 12),
                "flops": _FLOPS * n * t * case["scale"] ** p}
    if k in ("ids", "mask", "polys"):
        n = case["W"] * case["H"]
        return {"bytes": _scene_bytes(case["scene"]) + n * (4 if k == "ids" else 5),
                "flops": _FLOPS * n * _TILE_TESTS[case["scene"]] * (1 if k == "ids" else 2)}
    if k == "batch":
        b = f = 0.0
        for j in range(case["jobs"]):
            tris = max(200, int(case["tris"] * (j + 1) / case["jobs"]))
            size = case["size"] if j % 2 == 0 else max(33, case["size"] // 2 + 3)
            b += tris * 38 + size * size * 16
            f += _FLOPS * size * size * _TESTS["job"][0] * tris / 20000
        return {"bytes": b, "flops": f}
    if k == "kd":
        s = _scene(case["scene"])
        n = len(s.tris)
        return {"bytes": s.pos.nbytes + 12 * n + 28 * n + 60 * n, "flops": 50.0 * n * max(1.0, math.log2(n))}
    n = sum((case["size"] if j % 2 == 0 else case["size"] // 2 + 1) ** 2 for j in range(case["requests"]))
    return {"bytes": _scene_bytes("plant") + _scene_bytes("sphere5") + 10 * n, "flops": _FLOPS * 70.0 * n}


def tolerance(case):
    """Visibility and irradiance are sums of up to thousands of 32-bit clipped pieces: against
    64 bits they are 1e-7 to 1e-5 off (exact(), largest on a frame of the plant, where a few
    pixels at a leaf's edge see another light).  Ids, masks and trees are whole values or
    copied floats."""
    if case["kind"] in ("soft", "points", "batch", "serve"):
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.0}
    return "exact"


# ------------------------------------------------------- the result in 64 bits

def _clip(P, cnt, d, keep):
    """Part of each convex polygon P (m, V, 2) with `cnt` corners where d >= 0 (d: m, V; rows not in `keep` come out empty)."""
    m, V = d.shape
    i = torch.arange(V, device=P.device)[None, :]
    used = (i < cnt[:, None]) & keep[:, None]
    j = torch.where(i + 1 >= cnt[:, None], torch.zeros_like(i), i + 1).expand(m, V)
    dj = d.gather(1, j)
    Pj = P.gather(1, j[..., None].expand(m, V, 2))
    inside = used & (d >= 0)
    cross = used & ((d >= 0) != (dj >= 0))
    t = torch.where(cross, d / torch.where(cross, d - dj, torch.ones_like(d)), torch.zeros_like(d))
    X = P + t[..., None] * (Pj - P)
    emit = inside.long() + cross.long()
    at = emit.cumsum(1) - emit
    out = torch.zeros(m, V + 2, 2, dtype=P.dtype, device=P.device)
    row = torch.arange(m, device=P.device)[:, None].expand(m, V)
    a = inside & (at < V)
    out[row[a], at[a]] = P[a]
    at2 = at + inside.long()
    b = cross & (at2 < V)
    out[row[b], at2[b]] = X[b]
    n = emit.sum(1).clamp(max=V)
    return out[:, :V], torch.where(n >= 3, n, torch.zeros_like(n))


def _area(P, cnt):
    V = P.shape[1]
    i = torch.arange(V, device=P.device)[None, :]
    j = torch.where(i + 1 >= cnt[:, None], torch.zeros_like(i), i + 1).expand(P.shape[0], V)
    Q = P.gather(1, j[..., None].expand(*P.shape))
    a = P[..., 0] * Q[..., 1] - Q[..., 0] * P[..., 1]
    return 0.5 * torch.where(i < cnt[:, None], a, torch.zeros_like(a)).sum(1)


def _soft_exact(pos, tris, light, offset, tri, X, N, exact, limit=30_000_000):
    """vis, E and Eu of shading points by subtracting every occluder's shadow from the light polygon, in 64 bits."""
    dev = X.device
    f8 = torch.float64
    Tv = torch.as_tensor(pos.astype(np.float64), device=dev)[torch.as_tensor(tris.astype(np.int64), device=dev)]
    Lc, U, Vv = (torch.as_tensor(light[3 * k:3 * k + 3], dtype=f8, device=dev) for k in range(3))
    n = X.shape[0]
    nL = torch.linalg.cross(U, Vv)
    A = nL.norm()
    nL = nL / A
    w = Lc - X
    r2 = (w * w).sum(1)
    wn = w / r2.sqrt()[:, None]
    lit = ((X - Lc) @ nL > 0) & (tri >= 0)
    G0 = (N * wn).sum(1).clamp(min=0) * (-(wn @ nL)).clamp(min=0) / r2
    zero = torch.zeros(n, dtype=f8, device=dev)
    Eu = torch.where(lit, A * G0, zero)
    back = tri < 0
    # pieces of the light in (s, t), U and V units, above the horizon
    V = 14
    own = torch.nonzero(lit).ravel()
    m = own.numel()
    P = torch.zeros(m, V, 2, dtype=f8, device=dev)
    quad = torch.tensor([[-.5, -.5], [.5, -.5], [.5, .5], [-.5, .5]], dtype=f8, device=dev)
    P[:, :4] = quad
    cnt = torch.full((m,), 4, dtype=torch.long, device=dev)
    h = (N[own] * (Lc - X[own])).sum(1)[:, None] + P[..., 0] * (N[own] @ U)[:, None] + P[..., 1] * (N[own] @ Vv)[:, None]
    P, cnt = _clip(P, cnt, h, torch.ones(m, dtype=torch.bool, device=dev))
    sel = cnt > 0
    P, cnt, own = P[sel], cnt[sel], own[sel]
    O = X + offset * N
    # which triangles can reach the light polygon of which point
    pts, occ = [], []
    chunk = max(1, 8_000_000 // len(Tv))
    corner = Lc + quad[:, :1] * U + quad[:, 1:] * Vv
    total = 0

    def lines(p, t):
        """The four half planes of triangle t's shadow seen from point p, as coefficients of (1, s, u)."""
        r = [Tv[t, k] - O[p] for k in range(3)]
        mm = [torch.linalg.cross(r[k], r[(k + 1) % 3], dim=-1) for k in range(3)]
        nn = torch.linalg.cross(Tv[t, 1] - Tv[t, 0], Tv[t, 2] - Tv[t, 0], dim=-1)
        D = (r[2] * mm[0]).sum(-1)
        sg = torch.where(D > 0, 1.0, -1.0).to(f8)
        C = (nn * r[0]).sum(-1)
        sc = torch.where(C > 0, 1.0, -1.0).to(f8)
        d0 = Lc - O[p]
        out = [torch.stack([sg * (q * d0).sum(-1), sg * (q @ U), sg * (q @ Vv)], -1) for q in mm]
        out.append(torch.stack([sc * (nn * d0).sum(-1) - C.abs(), sc * (nn @ U), sc * (nn @ Vv)], -1))
        return torch.stack(out, -2), D.abs() > 1e-14 * mm[0].norm(dim=-1) * r[2].norm(dim=-1)

    live = torch.unique(own)
    ids = torch.arange(len(Tv), device=dev)
    for c in torch.split(live, chunk):
        p = c[:, None].expand(-1, len(Tv)).reshape(-1)
        t = ids[None, :].expand(len(c), -1).reshape(-1)
        L, ok = lines(p, t)
        best = torch.stack([L[..., 0] + L[..., 1] * q[0] + L[..., 2] * q[1] for q in quad], -1).amax(-1)
        ok &= (best > 0).all(-1) & (t != tri[p])
        p, t = p[ok], t[ok]
        # a side of the beam that has all three corners outside
        e = corner[None] - O[p][:, None]
        side = torch.linalg.cross(e, e[:, [1, 2, 3, 0]], dim=-1)
        side = side * torch.sign((side * e.mean(1, keepdim=True)).sum(-1, keepdim=True))
        s = torch.einsum("pkc,pvc->pkv", side, Tv[t] - O[p][:, None])
        ok = ~((s < 0).all(-1).any(-1))
        pts.append(p[ok])
        occ.append(t[ok])
        total += int(ok.sum())
        if total > limit:
            return None
    pts, occ = torch.cat(pts), torch.cat(occ)
    order = torch.argsort(pts, stable=True)
    pts, occ = pts[order], occ[order]
    count = torch.bincount(pts, minlength=n)
    start = count.cumsum(0) - count
    for k in range(int(count.max()) if total else 0):
        has = count[own] > k
        if not bool(has.any()):
            break
        sel = torch.nonzero(has).ravel()
        L, _ = lines(own[sel], occ[start[own[sel]] + k])
        d = L[:, :, 0, None] + L[:, :, 1, None] * P[sel, None, :, 0] + L[:, :, 2, None] * P[sel, None, :, 1]
        used = torch.arange(V, device=dev)[None, None, :] < cnt[sel][:, None, None]
        meets = ((d > 0) & used).any(-1).all(-1)
        sel, L = sel[meets], L[meets]
        if sel.numel() == 0:
            continue
        Q, c, o = P[sel], cnt[sel], own[sel]
        newP, newC, newO = [], [], []
        for e in range(4):
            d = L[:, e, 0, None] + L[:, e, 1, None] * Q[..., 0] + L[:, e, 2, None] * Q[..., 1]
            on = c > 0
            B, bc = _clip(Q, c, -d, on)
            g = (bc > 0) & (_area(B, bc).abs() > 1e-15)
            newP.append(B[g])
            newC.append(bc[g])
            newO.append(o[g])
            Q, c = _clip(Q, c, d, on)
        rest = torch.ones(len(own), dtype=torch.bool, device=dev)
        rest[sel] = False
        P, cnt, own = torch.cat([P[rest]] + newP), torch.cat([cnt[rest]] + newC), torch.cat([own[rest]] + newO)
        if len(own) > limit // 10:
            return None
    vis = zero.clone().index_add_(0, own, _area(P, cnt).abs()).clamp(0, 1)
    if exact:
        Y = Lc + P[..., :1] * U + P[..., 1:] * Vv - X[own][:, None]
        i = torch.arange(V, device=dev)[None, :]
        j = torch.where(i + 1 >= cnt[:, None], torch.zeros_like(i), i + 1).expand(len(own), V)
        Z = Y.gather(1, j[..., None].expand(-1, -1, 3))
        g = torch.linalg.cross(Y, Z, dim=-1)
        lg = g.norm(dim=-1)
        th = torch.atan2(lg, (Y * Z).sum(-1))
        term = torch.where((i < cnt[:, None]) & (lg > 0), th * (g * N[own][:, None]).sum(-1) / lg.clamp(min=1e-300),
                           torch.zeros_like(lg))
        E = zero.clone().index_add_(0, own, 0.5 * term.sum(1).abs())
    else:
        E = Eu * vis
    vis = torch.where(back, -torch.ones_like(vis), vis)
    return vis.cpu().numpy(), E.cpu().numpy(), Eu.cpu().numpy()


def _eye_hits(s, view, W, H, dev):
    """The nearest triangle, hit point and normal facing the eye through every pixel centre, in 64 bits by brute force."""
    f8 = torch.float64
    eye, target, up = (torch.as_tensor(np.asarray(a, np.float32).astype(np.float64), device=dev)
                       for a in (view[0], view[1], s.up))
    fwd = (target - eye) / (target - eye).norm()
    right = torch.linalg.cross(fwd, up)
    right = right / right.norm()
    down = torch.linalg.cross(fwd, right)
    hh = math.tan(view[2] * math.pi / 360)
    hw = hh * W / H
    x = (2 * (torch.arange(W, dtype=f8, device=dev) + .5) / W - 1) * hw
    y = (2 * (torch.arange(H, dtype=f8, device=dev) + .5) / H - 1) * hh
    D = (fwd + x[None, :, None] * right + y[:, None, None] * down).reshape(-1, 3)
    T = torch.as_tensor(s.pos.astype(np.float64), device=dev)[torch.as_tensor(s.tris.astype(np.int64), device=dev)]
    r = T - eye
    # det and barycentric numerators are linear in the direction
    e1, e2 = r[:, 1] - r[:, 0], r[:, 2] - r[:, 0]
    n = torch.linalg.cross(e1, e2)
    a1, a2 = torch.linalg.cross(r[:, 2], r[:, 0]), torch.linalg.cross(r[:, 0], r[:, 1])
    C = (n * r[:, 0]).sum(1)
    tri = torch.full((len(D),), -1, dtype=torch.long, device=dev)
    best = torch.full((len(D),), math.inf, dtype=f8, device=dev)
    for c in torch.split(torch.arange(len(D), device=dev), max(1, 40_000_000 // len(T))):
        d = D[c]
        det = d @ n.T
        t = C / det
        u, v = (d @ a1.T) / det, (d @ a2.T) / det
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (det != 0), t, torch.full_like(t, math.inf))
        b, k = t.min(1)
        best[c], tri[c] = b, torch.where(torch.isfinite(b), k, torch.full_like(k, -1))
    hit = tri >= 0
    X = torch.where(hit[:, None], eye + D * torch.where(hit, best, torch.zeros_like(best))[:, None], torch.zeros_like(D))
    N = n[tri.clamp(min=0)]
    N = N / N.norm(dim=1, keepdim=True)
    N = N * torch.where((N * D).sum(1) > 0, -1.0, 1.0)[:, None]
    return tri, X, N


def exact(case, seed):
    """By brute force over all pairs of points and triangles where that takes seconds: room and plant.
    Ids, masks and trees are whole values and have none."""
    if case["kind"] not in ("soft", "points") or case["scene"] not in ("room", "plant"):
        return None
    s, d = _scene(case["scene"]), _inputs(case, seed)
    dev = torch.device("cuda", 0)
    diag = np.float32(np.linalg.norm((s.pos.max(0) - s.pos.min(0)).astype(np.float64)))
    offset = float(diag * np.float32(2e-5))
    if case["kind"] == "soft":
        tri, X, N = _eye_hits(s, d["view"], case["W"], case["H"], dev)
    else:
        tri = torch.as_tensor(d["tri"].astype(np.int64), device=dev)
        X, N = (torch.as_tensor(d[k].astype(np.float64), device=dev) for k in "XN")
    got = _soft_exact(s.pos, s.tris, d["light"], offset, tri, X, N, case["exact"])
    if got is None:
        return None
    out = dict(zip(("vis", "E", "Eu"), got))
    if case["kind"] == "soft":
        out["tri"] = None
    return out
