"""The ray-query work that users of this library have it do, as cases to be timed.

A case is a dict of plain values.  ``listed()`` gives the named ones, ``draw``
one more of the same ranges, ``prepare`` what a program holds before the call
(trees on the device, rays, a camera, a plan), ``run`` one pass through the
public entry points and ``work`` the bytes and operations one pass cannot do
without.  Meshes are fixed assets, generated once per process; every
``prepare`` uploads them and builds its own trees, and the seed moves the
camera, the rays and the animation.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rfmanta_b200 import scenes
from rfmanta_b200.batch import BatchedQueries, QueryBatch
from rfmanta_b200.dynbvh import GpuDynBVH, InstancedBVH, RayBatch
from rfmanta_b200.serve import RenderServer, request_for_scene

WALD, KS = 0, 1
FAR = 64.0  # closest-hit rays end here (every scene's diagonal is below 16)


def listed():
    return [
        # one 64-ray packet of a render worker (DynBVH::intersect through the
        # host-array call): the smallest call there is, all latency
        {"name": "packet_closest_64", "what": "host_rays", "scene": "sphere", "size": 6,
         "rays": "camera", "n": 64, "anyhit": False, "tri": WALD},
        # a host program's own shadow test, a ragged batch past the packet
        # size: copies in and out, Kensler-Shirley triangles
        {"name": "host_anyhit_50021", "what": "host_rays", "scene": "heightfield", "size": 128,
         "rays": "random", "n": 50021, "anyhit": True, "tri": KS},
        # rays a simulation already has on the device: incoherent closest hit
        {"name": "device_closest_1m", "what": "device_rays", "scene": "heightfield", "size": 384,
         "rays": "random", "n": 1 << 20, "anyhit": False, "tri": WALD},
        # coherent camera rays from a caller's own camera model, odd count,
        # Kensler-Shirley
        {"name": "device_camera_ks", "what": "device_rays", "scene": "spheres", "size": 20,
         "rays": "camera", "n": 777_777, "anyhit": False, "tri": KS},
        # occlusion queries over a large scene
        {"name": "device_anyhit_3m", "what": "device_rays", "scene": "heightfield", "size": 640,
         "rays": "random", "n": 3_000_001, "anyhit": True, "tri": WALD},
        # the interactive frame: 512x512, one sample, one light
        {"name": "whitted_512", "what": "whitted", "size": 6, "grid": 100, "xres": 512,
         "yres": 512, "tri": WALD},
        # an animated mesh: tree update with rotations and one frame
        {"name": "animate_512", "what": "animate", "size": 6, "grid": 100, "xres": 512,
         "yres": 512, "rotate": True, "tri": WALD},
        # the large coherent frame: two-level scene, 1920x1080, 4 samples
        {"name": "frame_1080p", "what": "frame", "size": 512, "instances": 64, "level": 6,
         "xres": 1920, "yres": 1080, "spp": 4, "tri": WALD},
        # a preview of the path tracer, odd resolution, Kensler-Shirley
        {"name": "path_preview", "what": "path", "size": 128, "xres": 333, "yres": 251, "spp": 4,
         "depth": 3, "tri": KS},
        # the path-traced frame the benchmark times: 1280x720, 16 samples, 1.2M triangles
        {"name": "path_720p", "what": "path", "size": 512, "xres": 1280, "yres": 720, "spp": 16,
         "depth": 4, "tri": WALD},
        # many uneven batches over several resident scenes in one launch
        {"name": "batched_24", "what": "batch", "scenes": 4, "batches": 24, "most": 2_000_000,
         "tri": WALD},
        # a render server with a queue of mixed requests waiting
        {"name": "serve_12", "what": "serve", "scenes": 3, "requests": 12, "most": 1280,
         "tri": WALD},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["host_rays", "device_rays", "device_rays", "whitted", "animate", "frame",
                       "path", "path", "batch", "serve"])
    c = {"what": what, "tri": rng.choice([WALD, WALD, KS])}
    if what in ("host_rays", "device_rays"):
        c["scene"] = rng.choice(["heightfield", "spheres", "sphere"])
        c["size"] = {"heightfield": lambda: _log(rng, 48, 640), "spheres": lambda: _log(rng, 2, 20),
                     "sphere": lambda: rng.randint(4, 6)}[c["scene"]]()
        c["rays"] = rng.choice(["random", "camera"])
        c["n"] = _log(rng, 64, 300_000) if what == "host_rays" else _log(rng, 4_000, 3_000_000)
        c["anyhit"] = rng.random() < 0.5
    elif what in ("whitted", "animate"):
        c.update(size=rng.randint(4, 6), grid=_log(rng, 10, 120), xres=_log(rng, 200, 1920))
        c["yres"] = int(c["xres"] * rng.uniform(0.5, 1.0))
        if what == "animate":
            c["rotate"] = rng.random() < 0.6
    elif what == "frame":
        c.update(size=_log(rng, 64, 512), instances=_log(rng, 4, 100), level=rng.randint(4, 6),
                 xres=_log(rng, 320, 1920), spp=rng.choice([1, 4]))
        c["yres"] = int(c["xres"] * rng.uniform(0.5, 0.57))
    elif what == "path":
        c.update(size=_log(rng, 64, 400), xres=_log(rng, 160, 1280), spp=rng.choice([1, 4, 9]),
                 depth=rng.randint(1, 5))
        c["yres"] = int(c["xres"] * rng.uniform(0.5, 0.57))
    elif what == "batch":
        c.update(scenes=rng.randint(1, 4), batches=rng.randint(6, 30),
                 most=_log(rng, 50_000, 2_000_000))
    else:
        c.update(scenes=rng.randint(1, 3), requests=rng.randint(4, 16),
                 most=rng.choice([512, 1280]))
    return c


# ---------------------------------------------------------------- assets ----

@functools.lru_cache(maxsize=None)
def _mesh(kind, size):
    if kind == "heightfield":
        m = scenes.heightfield(size, size, 100, extent=6.0, y=0.0)
        m.materials = np.array([[0.7, 0.7, 0.7]], np.float32)
        return m
    if kind == "spheres":
        return scenes.sphere_set(size, 5, 102)
    return scenes.small_frame_scene(level=size).mesh


@functools.lru_cache(maxsize=None)
def _whitted(size, grid):
    return scenes.small_frame_scene(level=size, grid=grid)


@functools.lru_cache(maxsize=None)
def _path(size):
    return scenes.path_scene(hf_nx=size, hf_nz=2 * size)


@functools.lru_cache(maxsize=None)
def _frame(size, instances, level):
    return scenes.coherent_scene(hf_n=size, n_instances=instances, sphere_level=level)


# the batched and served scenes: 10,240 to 819,200 triangles
_RESIDENT = [("spheres", 2), ("heightfield", 128), ("heightfield", 384), ("heightfield", 640)]


def _tree(mesh, tri):
    b = GpuDynBVH(tri_kind=tri, device=0)
    b.setGroup(mesh)
    b.rebuild()
    return b


def _camera(cam, xres, yres, rng):
    """The scene's camera moved round the vertical axis and a little up or
    down, with the vertical field of view of the resolution."""
    a = rng.uniform(-0.6, 0.6)
    e = np.asarray(cam.eye, np.float64) - cam.lookat
    eye = (cam.lookat[0] + e[0] * math.cos(a) + e[2] * math.sin(a),
           cam.lookat[1] + e[1] + rng.uniform(-0.2, 0.2),
           cam.lookat[2] - e[0] * math.sin(a) + e[2] * math.cos(a))
    vfov = 2 * math.degrees(math.atan(math.tan(math.radians(30.0)) * yres / xres))
    return scenes.Camera(tuple(float(x) for x in eye), cam.lookat, cam.up, 60.0, vfov)


def _with(obj, **new):
    out = object.__new__(type(obj))
    out.__dict__.update(obj.__dict__)
    out.__dict__.update(new)
    return out


def _rays(case, mesh, seed):
    """(org, dir, tmax) on the device, rows x/y/z."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["n"]
    lo, hi = (torch.tensor(x, device="cuda").view(3, 1) for x in mesh.bounds())
    if case["rays"] == "random":
        o = lo + (hi - lo) * torch.rand(3, n, generator=g, device="cuda")
        d = torch.randn(3, n, generator=g, device="cuda")
    else:  # rows of an image, jittered, from a point above and in front
        w = max(8, int(math.sqrt(n * 16 / 9)))
        k = torch.arange(n, device="cuda")
        jit = torch.rand(2, n, generator=g, device="cuda")
        x = ((k % w) + jit[0]) / w * 2 - 1
        y = ((k // w) + jit[1]) / max(1, -(-n // w)) * 2 - 1
        ext = (hi - lo).max()
        side = torch.rand(1, generator=g, device="cuda") * 0.6 - 0.3
        c = (lo + hi) / 2
        eye = c + ext * torch.stack([side, side * 0 + 0.5, side * 0 + 1.0])
        f = (c - eye) / (c - eye).norm()
        up = torch.tensor([[0.0], [1.0], [0.0]], device="cuda")
        r = torch.linalg.cross(f, up, dim=0)
        u = torch.linalg.cross(r / r.norm(), f, dim=0)
        d = f + 0.58 * (x * r / r.norm() + y * u)
        o = eye.expand(3, n)
    d = d / d.norm(dim=0, keepdim=True)
    if case["anyhit"]:
        diag = float((hi - lo).norm())
        tmax = 0.1 + (diag - 0.1) * torch.rand(n, generator=g, device="cuda")
    else:
        tmax = torch.full((n,), FAR, device="cuda")
    return o.float().contiguous(), d.float().contiguous(), tmax


# --------------------------------------------------------------- prepare ----

def prepare(case, seed):
    what, tri = case["what"], case["tri"]
    rng = np.random.default_rng(seed)
    s = {"what": what}
    if what in ("host_rays", "device_rays"):
        mesh = _mesh(case["scene"], case["size"])
        o, d, tm = _rays(case, mesh, seed)
        s.update(bvh=_tree(mesh, tri), n=case["n"], anyhit=case["anyhit"])
        if what == "host_rays":
            s["rays"] = [x.cpu().numpy() for x in (o, d, tm)]
            s["flags"] = RayBatch.AnyHit if case["anyhit"] else 0
        else:
            s.update(o=o, d=d, tm=tm, t=torch.empty_like(tm), u=torch.empty_like(tm),
                     v=torch.empty_like(tm),
                     prim=torch.empty(case["n"], dtype=torch.int32, device="cuda"))
        return s
    if what in ("whitted", "animate"):
        sc = _whitted(case["size"], case["grid"])
        x, y = case["xres"], case["yres"]
        sc = _with(sc, camera=_camera(sc.camera, x, y, rng), xres=x, yres=y, mesh=_with(sc.mesh))
        s.update(bvh=_tree(sc.mesh, tri), params=GpuDynBVH.whitted_params(sc),
                 rgb=torch.empty(x * y, 3, device="cuda"), t=torch.empty(x * y, device="cuda"),
                 prim=torch.empty(x * y, dtype=torch.int32, device="cuda"),
                 count=torch.zeros(1, dtype=torch.int64, device="cuda"))
        if what == "animate":
            ph = rng.uniform(0, 2 * math.pi)
            v0 = sc.mesh.vertices
            s.update(k=0, rotate=case["rotate"], poses=[torch.from_numpy(np.ascontiguousarray(
                v0 + 0.01 * np.sin(3.0 * v0[:, [1, 2, 0]] + ph + 2 * math.pi * k / 8),
                np.float32)).cuda() for k in range(8)])
        return s
    if what == "frame":
        sc = _frame(case["size"], case["instances"], case["level"])
        x, y = case["xres"], case["yres"]
        sc = _with(sc, camera=_camera(sc.camera, x, y, rng), xres=x, yres=y, spp=case["spp"],
                   seed=int(seed))
        inner = [_tree(m, tri) for m in sc.inner]
        top = InstancedBVH(inner, sc.inst_scene, sc.translation, sc.kind)
        top.rebuild()
        s.update(bvh=top, inner=inner, params=GpuDynBVH.frame_params(sc, sc.materials),
                 rgb=torch.empty(x * y, 3, device="cuda"),
                 count=torch.zeros(1, dtype=torch.int64, device="cuda"))
        return s
    if what == "path":
        sc = _path(case["size"])
        x, y = case["xres"], case["yres"]
        sc = _with(sc, camera=_camera(sc.camera, x, y, rng), xres=x, yres=y, spp=case["spp"],
                   max_depth=case["depth"], seed=int(seed))
        s.update(bvh=_tree(sc.mesh, tri), params=GpuDynBVH.path_params(sc),
                 rgb=torch.empty(x * y, 3, device="cuda"),
                 count=torch.zeros(2, dtype=torch.int64, device="cuda"))
        return s
    meshes = [_mesh(k, n) for k, n in _RESIDENT[:case["scenes"]]]
    s["bvhs"] = [_tree(m, tri) for m in meshes]
    if what == "batch":
        # sizes spread over the logarithm from 1,000 rays up, half any hit:
        # the shape of the table is the case's, the rays are the seed's
        fixed = np.random.default_rng(7)
        batches = []
        for k in range(case["batches"]):
            n = int(math.exp(fixed.uniform(math.log(1000), math.log(case["most"]))))
            si, anyhit = int(fixed.integers(0, len(meshes))), bool(k % 2)
            o, d, tm = _rays({"n": n, "rays": "random", "anyhit": anyhit}, meshes[si],
                             int(rng.integers(0, 1 << 40)))
            batches.append(QueryBatch(si, o, d, tm, anyhit))
        s["plan"] = BatchedQueries(s["bvhs"], batches)
        return s
    stream = []
    for k in range(case["requests"]):
        x = [256, 512, 1280][k % (3 if case["most"] >= 1280 else 2)]
        y = 720 if x == 1280 else x
        si = k % len(meshes)
        stream.append((0.0, request_for_scene(si, meshes[si], x, y, [1, 4, 4, 16][k % 4] if
                                              x < 1280 else [1, 4][k % 2], [1, 3, 5][k % 3],
                                              int(seed) * 64 + k)))
    s.update(server=RenderServer(s["bvhs"], path_capacity=1 << 22, chunk_pixels=65536,
                                 hbm_budget_bytes=4 << 30), stream=stream)
    return s


# ------------------------------------------------------------------- run ----

def run(s):
    what = s["what"]
    if what == "host_rays":
        o, d, tm = s["rays"]
        r = RayBatch(o, d, tm, s["flags"])
        s["bvh"].intersect(r)
        return {"t": r.minT, "prim": r.hitPrim, "u": r.u, "v": r.v}
    if what == "device_rays":
        s["bvh"].intersect_device(s["n"], s["o"].data_ptr(), s["d"].data_ptr(),
                                  s["tm"].data_ptr(), s["anyhit"], s["t"].data_ptr(),
                                  s["prim"].data_ptr(), s["u"].data_ptr(), s["v"].data_ptr())
        return {"t": s["t"], "prim": s["prim"], "u": s["u"], "v": s["v"]}
    if what in ("whitted", "animate"):
        if what == "animate":
            s["bvh"].update_device(s["poses"][s["k"] % 8].data_ptr(), rotate=s["rotate"])
            s["k"] += 1
        s["bvh"].render_whitted_device(s["params"], s["rgb"].data_ptr(), s["t"].data_ptr(),
                                       s["prim"].data_ptr(), s["count"].data_ptr())
        return {"rgb": s["rgb"], "t": s["t"], "prim": s["prim"], "count": s["count"]}
    if what == "frame":
        s["bvh"].render_frame_device(s["params"], s["rgb"].data_ptr(), s["count"].data_ptr())
        return {"rgb": s["rgb"], "count": s["count"]}
    if what == "path":
        s["bvh"].render_path_device(s["params"], s["rgb"].data_ptr(), s["count"].data_ptr())
        return {"rgb": s["rgb"], "count": s["count"]}
    if what == "batch":
        s["plan"].launch()
        return {"t": s["plan"].t, "prim": s["plan"].prim}
    out = s["server"].run_stream(s["stream"], keep_images=True)
    return {"images": [out["info"][k]["image"] for k in range(len(s["stream"]))]}


# ------------------------------------------------------------ work, exact ----

def _tris(case):
    what = case["what"]
    if what in ("host_rays", "device_rays"):
        return {"heightfield": 2 * case["size"] ** 2, "spheres": 20480 * case["size"],
                "sphere": 20 * 4 ** case["size"] + 20000}[case["scene"]]
    if what in ("whitted", "animate"):
        return 20 * 4 ** case["size"] + 2 * case["grid"] ** 2
    if what == "frame":
        return 2 * case["size"] ** 2 + 20 * 4 ** case["level"]
    if what == "path":
        return 4 * case["size"] ** 2 + 32 * 5120
    return sum(20480 * n if k == "spheres" else 2 * n * n for k, n in _RESIDENT[:case["scenes"]])


def work(case):
    """Rays in and hits (or pixels) out once; of the scene, each triangle once
    or, for few rays, one root-to-leaf path of 32-byte boxes and a 48-byte
    triangle per ray; two box tests (24 operations each) per level of a
    balanced tree and one triangle test (40) per ray.  Frames: one camera ray
    per sample and one shadow ray per light or bounce on half of them."""
    what, tris = case["what"], _tris(case)
    io = 0
    if what in ("host_rays", "device_rays"):
        rays = case["n"]
        io = 28 * rays + 16 * rays
    elif what in ("whitted", "animate"):
        px = case["xres"] * case["yres"]
        rays, io = 1.5 * px, 20 * px
        if what == "animate":
            io += 36 * tris + 2 * 112 * tris  # positions and indices in, tree and records out
    elif what == "frame":
        px = case["xres"] * case["yres"]
        rays, io = 2 * px * case["spp"], 12 * px
    elif what == "path":
        px = case["xres"] * case["yres"]
        rays, io = 1.5 * px * case["spp"] * (1 + 0.5 * (case["depth"] - 1)), 12 * px
    elif what == "batch":
        fixed = np.random.default_rng(7)
        rays = 0
        for _ in range(case["batches"]):
            rays += int(math.exp(fixed.uniform(math.log(1000), math.log(case["most"]))))
            fixed.integers(0, case["scenes"])
        io = 28 * rays + 8 * rays
    else:
        rays = 0
        for k in range(case["requests"]):
            x = [256, 512, 1280][k % (3 if case["most"] >= 1280 else 2)]
            px = x * (720 if x == 1280 else x)
            spp = [1, 4, 4, 16][k % 4] if x < 1280 else [1, 4][k % 2]
            rays += 1.5 * px * spp * (1 + 0.5 * ([1, 3, 5][k % 3] - 1))
            io += 12 * px
    levels = math.log2(max(tris, 2))
    scene = min(18 * tris, rays * (32 * levels + 48))
    return {"bytes": io + scene, "flops": rays * (levels * 2 * 24 + 40)}


def _closest64(mesh, o, d, tmax):
    """Closest hit of every ray over every triangle in 64 bits (Moller and
    Trumbore): distance (tmax on a miss) and the hit's unit normal."""
    v = torch.from_numpy(mesh.vertices).cuda().double()
    i = torch.from_numpy(mesh.indices.astype(np.int64)).cuda()
    a, e1, e2 = v[i[:, 0]], v[i[:, 1]] - v[i[:, 0]], v[i[:, 2]] - v[i[:, 0]]
    best, which = tmax.double().clone(), torch.full_like(tmax, -1, dtype=torch.int64)
    step = max(1, (1 << 26) // a.shape[0])
    for r0 in range(0, o.shape[1], step):
        oo, dd = (x[:, r0:r0 + step].double().T[:, None, :] for x in (o, d))
        p = torch.linalg.cross(dd.expand(-1, a.shape[0], -1), e2[None].expand(dd.shape[0], -1, -1))
        inv = 1 / (p * e1).sum(-1)
        s = oo - a
        u = (s * p).sum(-1) * inv
        del p
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        w = (dd * q).sum(-1) * inv
        t = (e2 * q).sum(-1) * inv
        del q, s
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 1e-4), t, math.inf)
        m, k = t.min(dim=1)
        hit = m < best[r0:r0 + step]
        best[r0:r0 + step] = torch.where(hit, m, best[r0:r0 + step])
        which[r0:r0 + step] = torch.where(hit, k, -1)
    n = torch.linalg.cross(e1, e2)
    n = n / n.norm(dim=1, keepdim=True)
    return best, which, n


def exact(case, seed):
    """Closest-hit distances and one-sample frames by brute force in 64 bits;
    None where that takes too long, for an occluder's distance (any of them
    answers the query), for the triangles' own u and v, and for images built
    from random samples."""
    what = case["what"]
    if what in ("host_rays", "device_rays"):
        if case["anyhit"] or case["n"] * _tris(case) > 1.2e10:
            return None
        mesh = _mesh(case["scene"], case["size"])
        return {"t": _closest64(mesh, *_rays(case, mesh, seed))[0], "prim": None, "u": None,
                "v": None}
    if what != "whitted" or 2 * case["xres"] * case["yres"] * _tris(case) > 1.2e10:
        return None
    sc = _whitted(case["size"], case["grid"])
    x, y = case["xres"], case["yres"]
    cam = _camera(sc.camera, x, y, np.random.default_rng(seed))
    eye, at, up = (np.asarray(c, np.float32).astype(np.float64) for c in (cam.eye, cam.lookat,
                                                                         cam.up))
    f = at - eye
    side = np.cross(f, up / np.linalg.norm(up))
    side /= np.linalg.norm(side)
    top = np.cross(side, f)
    top /= np.linalg.norm(top)
    near = np.linalg.norm(f)
    side *= near * math.tan(math.radians(0.5 * np.float32(cam.hfov)))
    top *= near * math.tan(math.radians(0.5 * np.float32(cam.vfov)))
    px = ((np.arange(x) + 0.5) / x * 2 - 1)[None, :, None]
    py = ((np.arange(y) + 0.5) / y * 2 - 1)[:, None, None]
    d = (f + px * side + py * top).reshape(-1, 3)
    d = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).T.copy()).cuda()
    o = torch.from_numpy(eye).cuda().view(3, 1).expand_as(d)
    big = torch.full((x * y,), 1e19, device="cuda", dtype=torch.float64)
    t, which, n = _closest64(sc.mesh, o, d, big)
    hit = which >= 0
    nrm = n[which.clamp(min=0)].T
    nrm = torch.where((nrm * d).sum(0) <= 0, nrm, -nrm)
    p = o + d * torch.where(hit, t, 1.0)
    light = torch.tensor(sc.ambient, dtype=torch.float64, device="cuda").view(3, 1).repeat(1, x * y)
    for l in sc.lights:
        sd = torch.tensor(l.position, dtype=torch.float64, device="cuda").view(3, 1) - p
        front = hit & ((sd * nrm).sum(0) > 0)
        k = front.nonzero().view(-1)
        one = torch.full((k.numel(),), 1 - 1e-4, dtype=torch.float64, device="cuda")
        k = k[_closest64(sc.mesh, p[:, k], sd[:, k], one)[1] < 0]
        cos = (sd[:, k] * nrm[:, k]).sum(0) / sd[:, k].norm(dim=0)
        light[:, k] += torch.tensor(l.color, dtype=torch.float64, device="cuda").view(3, 1) * cos
    mats = torch.from_numpy(sc.mesh.materials).cuda().double()
    kd = mats[torch.from_numpy(sc.mesh.face_material.astype(np.int64)).cuda()[which.clamp(min=0)]].T
    bg = torch.tensor(sc.background, dtype=torch.float64, device="cuda").view(3, 1)
    return {"rgb": torch.where(hit, light * kd, bg).T.contiguous(), "t": None, "prim": None,
            "count": None}
