"""Performance cases: the work programs have this library do, through its
public entry points, from calls that are all latency to full-size scenes.

A case is a dict with a ``kind``:

* ``closest``  -- closest hits of a batch of rays (``Mbvh.intersect``) over a
  structure that the program built before;
* ``any_hit``  -- occlusion of shadow rays, same entry point;
* ``build``    -- ``Builder`` + ``Mbvh.construct`` over device triangles, with
  the host copies of the drop-in API (``mirror``) or device-only;
* ``refit``    -- one animation step: ``Bvh.refit`` from moved triangles with
  the re-collapse of its Mbvh;
* ``diff``     -- differentiable closest hit, forward and backward;
* ``batch``    -- many meshes built and traced by one captured graph.

Scenes: ``sphere`` (closed noisy lat-long sphere), ``soup`` (triangles of
log-normal size, uniform in the unit cube) and ``clustered`` (64 spheres of
log-uniform radii). All inputs come from torch generators seeded by ``seed``.
"""
import ctypes
import math

import numpy as np
import torch

import rtbvh_gb300 as rb
from rtbvh_gb300 import _ffi
from rtbvh_gb300.api import DeviceArray
from rtbvh_gb300.diff import ray_cast

DEV = "cuda"
FAR = 100.0  # far plane of the camera rays


def listed():
    return [
        # a low-resolution probe or a pick over a small model: launch latency
        {"name": "probe_sphere_6400", "kind": "closest", "scene": "sphere", "builder": "sah", "tris": 6400,
         "rays": "camera", "count": 4096},
        # primary rays of a 1024 x 1024 image of the same model
        {"name": "camera_sphere_6400", "kind": "closest", "scene": "sphere", "builder": "sah", "tris": 6400,
         "rays": "camera", "count": 1048576},
        # the headline workload: incoherent rays through a large soup
        {"name": "incoherent_soup_1m", "kind": "closest", "scene": "soup", "builder": "locb", "tris": 1000000,
         "rays": "incoherent", "count": 16777216},
        # path tracing: cosine-weighted rays that leave the surfaces of a large scene
        {"name": "secondary_clustered_2m", "kind": "closest", "scene": "clustered", "builder": "sah",
         "tris": 2000003, "rays": "surface", "count": 4000037},
        # shadow rays from the surfaces of a scene towards a light
        {"name": "shadow_clustered_1m", "kind": "any_hit", "scene": "clustered", "builder": "locb",
         "tris": 1000000, "rays": "shadow", "count": 4194304},
        # drop-in use: a small model built with host copies of the nodes
        {"name": "build_locb_6400_mirror", "kind": "build", "scene": "sphere", "builder": "locb", "tris": 6400,
         "mirror": True},
        # a small model rebuilt for the GPU traversal, the SAH builder
        {"name": "build_sah_6400", "kind": "build", "scene": "sphere", "builder": "sah", "tris": 6400,
         "mirror": False},
        # a large scene, fast builder
        {"name": "build_locb_1m", "kind": "build", "scene": "soup", "builder": "locb", "tris": 1000000,
         "mirror": False},
        # a very large scene, quality builder
        {"name": "build_sah_clustered_4m", "kind": "build", "scene": "clustered", "builder": "sah",
         "tris": 4000000, "mirror": False},
        # one frame of an animated mesh
        {"name": "refit_sphere_200k", "kind": "refit", "scene": "sphere", "builder": "locb", "tris": 200000},
        # one gradient step of a mesh fit against a 2048 x 2048 image
        {"name": "diff_sphere_200k", "kind": "diff", "scene": "sphere", "builder": "locb", "tris": 200000,
         "rays": "camera", "count": 4194304},
        # a data set of meshes, each built and traced with rays of its own
        {"name": "batch_64_meshes", "kind": "batch", "meshes": 64, "lo": 64, "hi": 200000},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "closest", "any_hit", "build", "build", "build", "build", "refit",
                       "diff", "batch"])
    if kind == "closest":
        scene, rays = rng.choice([("sphere", "camera"), ("soup", "incoherent"), ("clustered", "surface")])
        return {"kind": kind, "scene": scene, "builder": rng.choice(["locb", "sah"]),
                "tris": _log_int(rng, 1000, 2000000), "rays": rays, "count": _log_int(rng, 4000, 8000000)}
    if kind == "any_hit":
        return {"kind": kind, "scene": "clustered", "builder": rng.choice(["locb", "sah"]),
                "tris": _log_int(rng, 5000, 1000000), "rays": "shadow", "count": _log_int(rng, 4000, 4000000)}
    if kind == "build":
        scene = rng.choice(["sphere", "soup", "clustered"])
        tris = _log_int(rng, 1000, 4000000)
        return {"kind": kind, "scene": scene, "builder": rng.choice(["locb", "sah"]), "tris": tris,
                "mirror": tris < 20000 and rng.random() < 0.5}
    if kind == "refit":
        return {"kind": kind, "scene": "sphere", "builder": rng.choice(["locb", "sah"]),
                "tris": _log_int(rng, 5000, 1000000)}
    if kind == "diff":
        return {"kind": kind, "scene": "sphere", "builder": rng.choice(["locb", "sah"]),
                "tris": _log_int(rng, 2000, 400000), "rays": "camera", "count": _log_int(rng, 16000, 4000000)}
    return {"kind": kind, "meshes": rng.randint(4, 64), "lo": 64, "hi": _log_int(rng, 2000, 200000)}


# ------------------------------------------------------------------ scenes and rays
def _generator(seed, what):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + what) & 0x7FFFFFFF)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _sphere(g, tris, radius=1.0):
    """At least `tris` triangles of a closed lat-long sphere, cut to `tris`."""
    n_lat = max(2, int(round(math.sqrt(tris / 4.0))))
    n_lon = max(3, -(-tris // (2 * n_lat)))
    fac = 0.95 + 0.1 * _uniform(g, n_lat + 1, n_lon)
    fac[0] = fac[0, 0]
    fac[-1] = fac[-1, 0]
    theta = torch.arange(n_lat + 1, device=DEV, dtype=torch.float64)[:, None] * (math.pi / n_lat)
    phi = torch.arange(n_lon, device=DEV, dtype=torch.float64)[None, :] * (2.0 * math.pi / n_lon)
    sin = torch.sin(theta)
    sin[0] = 0.0
    sin[-1] = 0.0
    p = torch.stack([sin * torch.cos(phi), sin * torch.sin(phi), torch.cos(theta).expand(-1, n_lon)], -1)
    p = p * (radius * fac)[..., None]
    q = torch.roll(p, -1, dims=1)
    a, b, d, e = p[:-1], q[:-1], p[1:], q[1:]
    t = torch.stack([torch.stack([a, d, e], -2), torch.stack([a, e, b], -2)], 2)
    return t.reshape(-1, 3, 3)[:tris]


def _soup(g, tris):
    c = _uniform(g, tris, 1, 3)
    length = 0.005 * torch.exp(0.5 * _normal(g, tris, 3, 1))
    return c + _unit(_normal(g, tris, 3, 3)) * length


def _clustered(g, tris):
    """64 spheres, radii log-uniform in [0.01, 0.2], centres from a
    4-component Gaussian mixture; triangles shared out by area."""
    radii = torch.exp(math.log(0.01) + math.log(20.0) * _uniform(g, 64))
    means = -0.6 + 1.2 * _uniform(g, 4, 3)
    comp = torch.randint(0, 4, (64,), generator=g, device=DEV)
    centres = (means[comp] + 0.25 * _normal(g, 64, 3)).clamp(-1.0, 1.0)
    share = (radii ** 2 / (radii ** 2).sum()).tolist()
    counts = [max(8, int(tris * s)) for s in share]
    counts[counts.index(max(counts))] += tris - sum(counts)
    parts = [_sphere(g, n, r) + c for n, r, c in zip(counts, radii.tolist(), centres)]
    return torch.cat(parts)


def _scene(case, seed):
    g = _generator(seed, 1)
    make = {"sphere": _sphere, "soup": _soup, "clustered": _clustered}[case["scene"]]
    return make(g, case["tris"]).to(torch.float32).contiguous()


def _camera(g, count):
    """Pinhole camera at distance 3 in a seeded direction, looking at the
    origin: the first `count` pixels of the smallest square image."""
    w = math.isqrt(count - 1) + 1
    back = _unit(_normal(g, 3))
    up = torch.zeros(3, device=DEV, dtype=torch.float64)
    up[int(back.abs().argmin())] = 1.0
    right = _unit(torch.linalg.cross(up, back))
    up = torch.linalg.cross(back, right)
    k = torch.arange(count, device=DEV)
    s = math.tan(math.radians(45.0) * 0.5)
    x = (((k % w) + 0.5) / w * 2.0 - 1.0) * s
    y = (1.0 - ((k // w) + 0.5) / w * 2.0) * s
    d = _unit(x[:, None] * right + y[:, None] * up - back)
    return torch.cat([(3.0 * back).expand(count, 3), d], 1), torch.full((count,), FAR, device=DEV)


def _incoherent(g, count):
    o = 0.5 + 2.0 * _unit(_normal(g, count, 3))
    return torch.cat([o, _unit(_uniform(g, count, 3) - o)], 1), None


def _surface_points(g, tris, count):
    """Points on random triangles, 1e-4 off the surface, and their normals."""
    t = tris[torch.randint(0, tris.shape[0], (count,), generator=g, device=DEV)].double()
    a, b = _uniform(g, count, 1), _uniform(g, count, 1)
    s = torch.sqrt(a)
    n = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-30)
    return (1.0 - s) * t[:, 0] + s * (1.0 - b) * t[:, 1] + s * b * t[:, 2] + 1e-4 * n, n


def _surface(g, tris, count):
    p, n = _surface_points(g, tris, count)
    d = n + 0.999 * _unit(_normal(g, count, 3))  # cosine-weighted around the normal
    return torch.cat([p, _unit(d)], 1), None


def _shadow(g, tris, count):
    p, _ = _surface_points(g, tris, count)
    to = 2.0 * _unit(_normal(g, 3)) + 0.05 * _normal(g, count, 3) - p
    dist = to.norm(dim=1, keepdim=True)
    return torch.cat([p, to / dist], 1), (0.999 * dist[:, 0]).to(torch.float32)


def _rays(case, seed, tris):
    g = _generator(seed, 2)
    kind, count = case["rays"], case["count"]
    if kind == "camera":
        rays, far = _camera(g, count)
    elif kind == "incoherent":
        rays, far = _incoherent(g, count)
    elif kind == "surface":
        rays, far = _surface(g, tris, count)
    else:
        rays, far = _shadow(g, tris, count)
    return rays.to(torch.float32).contiguous(), far


def _upstream(seed, count):
    return torch.randn(3, count, generator=_generator(seed, 3), device=DEV)


def _meshes(case, seed):
    """Vertices, rays and their offsets: spheres of log-uniform triangle
    counts around scattered centres, round(2000 sqrt(n)) rays each."""
    g = _generator(seed, 4)
    m = case["meshes"]
    u = [((7 * k) % m + 0.5) / m if m % 7 else (k + 0.5) / m for k in range(m)]
    centres = -5.0 + 10.0 * _uniform(g, m, 3)
    tris, rays, prim_offsets, ray_offsets = [], [], [0], [0]
    for x, c in zip(u, centres):
        n = int(math.exp(math.log(case["lo"]) + x * math.log(case["hi"] / case["lo"])))
        r = int(round(2000.0 * math.sqrt(n)))
        o = 2.0 * _unit(_normal(g, r, 3))
        d = _unit(-1.0 + 2.0 * _uniform(g, r, 3) - o)
        tris.append(_sphere(g, n) + c)
        rays.append(torch.cat([o + c, d], 1))
        prim_offsets.append(prim_offsets[-1] + n)
        ray_offsets.append(ray_offsets[-1] + r)
    return (torch.cat(tris).to(torch.float32).contiguous(), torch.cat(rays).to(torch.float32).contiguous(),
            prim_offsets, ray_offsets)


def _build(tris, builder, mirror=False):
    b = rb.Builder(primitives=rb.Triangles(tris))
    bvh = (b.construct_locally_ordered_clustered(host_mirror=mirror) if builder == "locb"
           else b.construct_binned_sah(host_mirror=mirror))
    return bvh, rb.Mbvh.construct(bvh, host_mirror=mirror)


# ------------------------------------------------------------------ the measured calls
def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "batch":
        v, r, po, ro = _meshes(case, seed)
        state["batch"] = rb.Batch(v, po, r, ro)
        return state
    tris = _scene(case, seed)
    state["tris"] = tris
    if case["kind"] in ("build", "refit"):
        n = case["tris"]
        shapes = {"nodes": (2 * n, 8), "indices": (n,), "quads": (n, 32)}
        if case.get("mirror"):
            state["out"] = {k: np.zeros(shape, "i4") for k, shape in shapes.items()}
        else:
            state["out"] = {k: torch.zeros(shape, dtype=torch.int32, device=DEV) for k, shape in shapes.items()}
    if case["kind"] == "build":
        return state
    state["bvh"], state["mbvh"] = _build(tris, case["builder"])
    if case["kind"] == "refit":
        step = 0.01 * torch.sin(3.0 * tris + 0.1 * torch.randn(1, 1, 3, generator=_generator(seed, 5), device=DEV))
        state["moved"] = (tris + step).contiguous()
        return state
    state["rays"], state["far"] = _rays(case, seed, tris)
    if case["kind"] == "diff":
        state["tris"].requires_grad_(True)
        state["rays"].requires_grad_(True)
        state["up"] = _upstream(seed, case["count"])
    return state


def _hits(hits):
    return {"t": hits[:, 0], "uv": hits[:, 1:3], "prim": hits.view(torch.int32)[:, 3]}


def _device_view(owner, is_mbvh, words):
    """Node and index arrays of a structure in device memory, as 32-bit words."""
    view = _ffi.RTGpuView()
    code = rb.load_library().rtbvh_gpu_view(owner.handle.id, is_mbvh, ctypes.byref(view))
    if code != rb.ResultCode.Ok:
        raise RuntimeError("rtbvh_gpu_view: %s" % code)
    return [torch.as_tensor(DeviceArray(ptr, shape, "<i4"), device=DEV)
            for ptr, shape in ((view.nodes, (view.node_count, words)), (view.indices, (view.index_count,)))]


def _keep(state, bvh, mbvh):
    """Copies a structure into the program's own arrays, as one with a
    renderer of its own does (node counts depend on the scene: the arrays
    have the largest size, the rest stays zero)."""
    nodes, indices = _device_view(bvh, 0, 8)
    quads = _device_view(mbvh, 1, 32)[0]
    out = state["out"]
    out["nodes"][:nodes.shape[0]].copy_(nodes)
    out["indices"].copy_(indices)
    out["quads"][:quads.shape[0]].copy_(quads)
    return out


def _keep_host(state, bvh, mbvh):
    """The same from the host copies."""
    nodes, quads = bvh.nodes().view("i4"), mbvh.quad_nodes().view("i4")
    out = state["out"]
    out["nodes"][:len(nodes)] = nodes
    out["indices"][:] = bvh.indices()
    out["quads"][:len(quads)] = quads
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("closest", "any_hit"):
        hits, _ = state["mbvh"].intersect(state["rays"], t_max=state["far"], any_hit=kind == "any_hit")
        return _hits(hits)
    if kind == "build":
        bvh, mbvh = _build(state["tris"], case["builder"], case["mirror"])
        return (_keep_host if case["mirror"] else _keep)(state, bvh, mbvh)
    if kind == "refit":
        state["bvh"].refit(triangles=state["moved"], mbvh=state["mbvh"])
        return _keep(state, state["bvh"], state["mbvh"])
    if kind == "diff":
        t, u, v, prim = ray_cast(state["mbvh"], state["tris"], state["rays"])
        up = state["up"]
        gv, gr = torch.autograd.grad((t, u, v), (state["tris"], state["rays"]), (up[0], up[1], up[2]))
        return {"t": t.detach(), "u": u.detach(), "v": v.detach(), "prim": prim, "grad_tris": gv, "grad_rays": gr}
    return _hits(state["batch"].run())


# ------------------------------------------------------------------ what a pass cannot do without
def _trace_work(tris, rays):
    """Each ray in (24 bytes) and its hit out (16), each triangle once; per
    ray the boxes on one way down a 4-wide tree and one triangle test."""
    depth = math.log(max(tris, 4)) / math.log(4.0)
    return 40.0 * rays + 36.0 * tris, rays * (depth * 4 * 20 + 60)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        span = math.log(case["hi"] / case["lo"])
        n = (case["hi"] - case["lo"]) / span  # means of the log-uniform sizes
        r = 2000.0 * 2.0 * (math.sqrt(case["hi"]) - math.sqrt(case["lo"])) / span
        b, f = _trace_work(n, r)
        return {"bytes": case["meshes"] * (b + 100.0 * n), "flops": case["meshes"] * (f + 200.0 * n)}
    n = case["tris"]
    if kind == "build":  # triangles in, 32-byte nodes, indices and 128-byte quad nodes out
        return {"bytes": n * (36.0 + 64.0 + 4.0 + 64.0), "flops": n * 200.0}
    if kind == "refit":
        return {"bytes": n * (36.0 + 64.0 + 64.0), "flops": n * 30.0}
    b, f = _trace_work(n, case["count"])
    if kind == "any_hit" or case["rays"] == "camera":
        b += 4.0 * case["count"]
    if kind == "diff":  # upstream gradients in, triangle and ray gradients out
        b += case["count"] * (12.0 + 24.0) + 36.0 * n
        f += case["count"] * 150.0
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values
EXACT_PAIRS = 1.0e10  # ray-triangle pairs that brute force does in a few seconds


def _test(o, d, v0, v1, v2):
    """Moeller-Trumbore: det, t, u, v (broadcast over leading dimensions)."""
    e1, e2 = v1 - v0, v2 - v0
    h = torch.linalg.cross(d, e2)
    det = (e1 * h).sum(-1)
    f = 1.0 / torch.where(det.abs() < 1e-5, torch.ones_like(det), det)
    s = o - v0
    q = torch.linalg.cross(s, e1)
    return det, f * (e2 * q).sum(-1), f * (s * h).sum(-1), f * (d * q).sum(-1)


def _nearest(tris, rays, far):
    """Index of each ray's nearest triangle, -1 for none."""
    tri = tris.double()
    v0, v1, v2 = tri[None, :, 0], tri[None, :, 1], tri[None, :, 2]
    best = []
    step = max(1, int(2.0e7 // tri.shape[0]))
    for k in range(0, rays.shape[0], step):
        r = rays[k:k + step].double()
        o, d = torch.broadcast_tensors(r[:, None, :3], v0)[0], torch.broadcast_tensors(r[:, None, 3:], v0)[0]
        det, t, u, v = _test(o, d, *torch.broadcast_tensors(v0, v1, v2))
        limit = far[k:k + step, None].double() if far is not None else 1e34
        ok = (det.abs() >= 1e-5) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-4) & (t < limit)
        t, i = torch.where(ok, t, torch.full_like(t, math.inf)).min(dim=1)
        best.append(torch.where(torch.isinf(t), torch.full_like(i, -1), i))
    return torch.cat(best)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("closest", "diff") or float(case["tris"]) * case["count"] > EXACT_PAIRS:
        return None
    tris = _scene(case, seed)
    rays, far = _rays(case, seed, tris)
    if kind == "diff":
        far = None
    with torch.no_grad():
        prim = _nearest(tris, rays, far)
    hit = prim >= 0
    v = tris.double().requires_grad_(True)
    r = rays.double().requires_grad_(True)
    tri = v[prim.clamp_min(0)]
    _, t, a, b = _test(r[:, :3], r[:, 3:], tri[:, 0], tri[:, 1], tri[:, 2])
    zero = torch.zeros_like(t)
    miss = far.double() if far is not None else torch.full_like(t, 1e34)
    out_t, out_u, out_v = torch.where(hit, t, miss), torch.where(hit, a, zero), torch.where(hit, b, zero)
    if kind == "closest":
        return {"t": out_t.detach(), "uv": torch.stack([out_u, out_v], 1).detach(), "prim": None}
    gv, gr = torch.autograd.grad((out_t, out_u, out_v), (v, r), tuple(_upstream(seed, case["count"]).double()))
    return {"t": out_t.detach(), "u": out_u.detach(), "v": out_v.detach(), "prim": None, "grad_tris": gv,
            "grad_rays": gr}
