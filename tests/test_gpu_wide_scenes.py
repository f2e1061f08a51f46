"""Scenes and rays that the wide walk (rq_wide.cuh) must take at the binary walk's
speed or better, and with its bits: far from the world's origin, with detail far
finer than the whole, along axes and in the planes of the boxes."""
import numpy as np
import pytest

from test_gpu_wide import _bits, _grid, _soup

pytestmark = pytest.mark.gpu


def _plan_pair(bvh, o, d, t, anyhit):
    """A default plan and the binary walk's (register stack entries)."""
    import torch
    from rfmanta_b200.batch import BatchedQueries, QueryBatch
    dev = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (o, d, t)]
    return [BatchedQueries([bvh], [QueryBatch(0, *dev, anyhit, want_uv=True)], cfg)
            for cfg in (None, dict(reg_stack=1))]


def _same_hits(bvh, o, d, t):
    import torch
    from rfmanta_b200.dynbvh import RayBatch
    for anyhit in (False, True):
        plans = _plan_pair(bvh, o, d, t, anyhit)
        for p in plans:
            p.launch()
        torch.cuda.synchronize()
        wide, binary = ([x[0].cpu().numpy() for x in (p.t, p.prim, p.u, p.v)] for p in plans)
        r = RayBatch(o, d, t, flags=RayBatch.AnyHit if anyhit else 0)
        bvh.intersect(r)
        for a in (wide, [r.minT, r.hitPrim, r.u, r.v]):
            assert np.array_equal(a[1], binary[1])
            for i in (0, 2, 3):
                assert np.array_equal(_bits(a[i]), _bits(binary[i]))
        for p in plans:
            p.close()
    return int((binary[1] >= 0).sum())


def _times(plans, reps=7):
    import torch
    out = []
    for p in plans:
        ms = []
        for k in range(reps + 2):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            p.launch(torch.cuda.current_stream().cuda_stream)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        out.append(sorted(ms[2:])[reps // 2])
    return out


def _built(mesh, kind=0):
    from rfmanta_b200.dynbvh import GpuDynBVH
    b = GpuDynBVH(tri_kind=kind)
    b.setGroup(mesh)
    b.rebuild()
    return b


def _room_with_a_fine_sphere(radius):
    from rfmanta_b200 import scenes
    from rfmanta_b200.scenes import Mesh
    v, f = scenes.icosphere(6)
    room = np.array([[-3, -3, -3], [3, -3, -3], [3, 3, 3], [-3, 3, 3]], np.float64)
    k = v.shape[0]
    f = np.concatenate([f, [[k, k + 1, k + 2], [k, k + 2, k + 3]]]).astype(np.uint32)
    return Mesh(np.concatenate([v * radius + 0.4, room]).astype(np.float32), f,
                np.zeros(f.shape[0], np.uint32), np.full((1, 3), 0.5, np.float32))


@pytest.mark.parametrize("case", ["off 100", "off 1000", "fine 3e-3", "fine 1e-3"])
def test_far_and_fine_scenes_cost_what_others_do(case):
    """The boxes' padding follows the ray, not the coordinates: within a factor of
    two of the binary walk (the two differ by 0.7-0.9 near the origin; padding by
    the coordinate cost 7 to 200 times here)."""
    from rfmanta_b200 import scenes
    rng = np.random.default_rng(5)
    n = 1 << 17
    if case.startswith("off"):
        mesh = scenes.heightfield(256, 256, 7, extent=6.0)
        mesh.vertices = (mesh.vertices.astype(np.float64) +
                         [6.0 * float(case[4:]), 0.0, 2.0 * float(case[4:])]).astype(np.float32)
        lo, hi = (x.astype(np.float64) for x in mesh.bounds())
        o = lo + (hi - lo) * rng.random((n, 3))
        d = rng.normal(size=(n, 3))
    else:
        mesh = _room_with_a_fine_sphere(float(case[5:]))
        o = np.broadcast_to([-2.5, 2.0, 2.8], (n, 3))
        d = mesh.vertices[rng.integers(0, mesh.vertices.shape[0] - 4, n)].astype(np.float64) - o
    b = _built(mesh)
    t = np.full(n, 1e19, np.float32)
    assert _same_hits(b, o.T, d.T, t) > n // 4
    plans = _plan_pair(b, o.T, d.T, t, False)
    wide, binary = _times(plans)
    assert wide < 2 * binary, (wide, binary)
    for p in plans:
        p.close()
    b.close()


def _along_axes(mesh, seed, n=20000):
    """Rays with one or two zero components (either sign, and components too small
    to matter), origins exactly in the planes of the boxes and beside them, and
    rays just outside the wide walk's slope and distance."""
    rng = np.random.default_rng(seed)
    v = mesh.vertices.astype(np.float64)
    ext = max(float(np.ptp(v, axis=0).max()), 1e-3)
    target = v[rng.integers(0, v.shape[0], n)]
    mixed = rng.random((n, 1))
    target = np.where(rng.random((n, 1)) < 0.5, target,
                      mixed * target + (1 - mixed) * v[rng.integers(0, v.shape[0], n)])
    d = rng.normal(size=(n, 3))
    zero = rng.random((n, 3)) < 0.5
    d = np.where(zero, rng.choice([0.0, -0.0, 1e-30, -1e-18], (n, 3)), d)
    d[: n // 8] = rng.normal(size=(n // 8, 3)) * 10.0 ** -rng.uniform(0, 9, (n // 8, 3))
    far = ext * np.where(rng.random((n, 1)) < 0.1, 1e4, rng.uniform(0, 3, (n, 1)))
    o = target - d * far
    o = np.where(np.abs(d) < 1e-12, target, o)  # in the plane of the target, exactly
    t = rng.choice([1e19, np.inf, 3.0 * ext], n)
    return [np.ascontiguousarray(x, np.float32) for x in (o.T, d.T, t)]


def _boxes(n, seed):
    """Faces of boxes at whole coordinates: planes shared by many nodes."""
    from rfmanta_b200.scenes import Mesh
    rng = np.random.default_rng(seed)
    p = rng.integers(-6, 6, (n, 3))
    q = p + rng.integers(0, 4, (n, 3))
    tris = []
    for a, b in zip(p, q):
        k = int(rng.integers(0, 3))
        u, w = (k + 1) % 3, (k + 2) % 3
        c = np.array([a, a, a, a], np.float32)
        c[1, u] = c[2, u] = b[u]
        c[2, w] = c[3, w] = b[w]
        tris += [c[[0, 1, 2]], c[[0, 2, 3]]]
    v = np.concatenate(tris)
    return Mesh(v, np.arange(v.shape[0], dtype=np.uint32).reshape(-1, 3),
                np.zeros(2 * n, np.uint32), np.full((1, 3), 0.5, np.float32))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("name", ["grid", "boxes", "soup", "far grid"])
def test_rays_along_axes_and_in_the_boxes_planes(name, kind):
    mesh = {"grid": lambda: _grid(24), "boxes": lambda: _boxes(400, 3),
            "soup": lambda: _soup(500, 4),
            "far grid": lambda: _grid(16, scale=0.25, offset=(4096.0, -512.0, 0.5))}[name]()
    b = _built(mesh, kind)
    for seed in (1, 2, 3):
        assert _same_hits(b, *_along_axes(mesh, seed)) > 500
    b.close()


@pytest.mark.parametrize("case", ["vertical", "in planes", "along axes"])
def test_rays_along_axes_cost_what_others_do(case):
    """Below the binary walk, as other rays are (0.64-0.74 of it; the exact walk with
    a stack in local memory, a whole ray at a time, cost 1.12-1.27)."""
    from rfmanta_b200 import scenes
    mesh = scenes.heightfield(256, 256, 7, extent=6.0)
    rng = np.random.default_rng(6)
    n = 1 << 20
    lo, hi = (x.astype(np.float64) for x in mesh.bounds())
    o = lo + (hi - lo) * rng.random((n, 3))
    d = rng.normal(size=(n, 3))
    if case == "vertical":
        o[:, 1] = hi[1] + 1.0
        d[:] = [0.0, -1.0, 0.0]
    elif case == "in planes":
        d[:, 1] = 0.0
    else:
        d = np.eye(3)[rng.integers(0, 3, n)]
    b = _built(mesh)
    plans = _plan_pair(b, o.T, d.T, np.full(n, 1e19, np.float32), False)
    wide, binary = _times(plans)
    assert wide < 0.95 * binary, (wide, binary)
    for p in plans:
        p.close()
    b.close()


def _walks_wide(scene=None, plan=None):
    import ctypes as C
    from rfmanta_b200 import _lib
    w = C.c_int(-1)
    if plan is not None:
        _lib.check(_lib.lib.rq_batch_plan_walks_wide(plan._plan, C.byref(w)))
    else:
        _lib.check(_lib.lib.rq_scene_walks_wide(scene.handle, C.byref(w)))
    return bool(w.value)


def _far(mesh):
    mesh.vertices = (mesh.vertices + np.float32(1e4)).astype(np.float32)
    return mesh


@pytest.mark.parametrize("name", ["one", "two", "three", "five", "soup", "flat", "small far away",
                                  "doubled", "sphere", "heightfield", "far", "fine"])
def test_which_trees_are_walked_wide(name):
    """Every tree of more than one leaf, after a build and after each update, and
    the default plan over it; the comparisons of test_gpu_wide.py compare two
    walks only if this holds."""
    from test_gpu_wide import _meshes
    mesh = dict(_meshes()).get(name) or {"far": lambda: _far(_grid(9)),
                                         "fine": lambda: _room_with_a_fine_sphere(1e-3)}[name]()
    b = _built(mesh)
    o = np.zeros((3, 8), np.float32)
    plans = _plan_pair(b, o, o + 1, np.ones(8, np.float32), False)
    many = b.info().n_records > 0
    assert many == (name != "one")
    assert _walks_wide(b) == many
    assert [_walks_wide(plan=p) for p in plans] == [many, False]
    for rotate in (True, False, True) if many else ():
        mesh.vertices = (mesh.vertices * np.float32(1.01)).astype(np.float32)
        b.update(rotate=rotate)
        assert _walks_wide(b) == (b.info().n_records > 0)
        for p in plans:
            p.launch()
        assert [_walks_wide(plan=p) for p in plans] == [b.info().n_records > 0, False]
    for p in plans:
        p.close()
    b.close()


def test_a_plan_follows_its_scene_to_the_records_and_back():
    """Boxes that are not nested send scene and plan to the binary walk; the next
    tree brings both back."""
    import torch
    from rfmanta_b200.treeio import parse_dynbvh_blob
    mesh = _soup(300, 9)
    b = _built(mesh)
    blob = b.exportBlob()
    t = parse_dynbvh_blob(blob, mesh.n_tris)
    inner = np.nonzero((t.children == 0) & (np.arange(t.children.shape[0]) > 0))[0]
    for i in inner[:20]:
        c = (t.bounds[i, :3] + t.bounds[i, 3:]) / 2
        t.bounds[i] = np.concatenate([c, c]) + 0.4 * (t.bounds[i] - np.concatenate([c, c]))
    o, d, tmax = _along_axes(mesh, 3, 4000)
    p = _plan_pair(b, o, d, tmax, False)
    p[1].close()
    p = p[0]
    p.launch()
    torch.cuda.synchronize()
    want = p.prim[0].cpu().numpy()
    assert _walks_wide(b) and _walks_wide(plan=p)
    b.importTree(t)
    p.launch()
    assert not _walks_wide(b) and not _walks_wide(plan=p)
    b.importBlob(blob)
    p.launch()
    torch.cuda.synchronize()
    assert _walks_wide(b) and _walks_wide(plan=p)
    assert np.array_equal(p.prim[0].cpu().numpy(), want)
    p.close()
    b.close()


@pytest.mark.parametrize("case,wide", [("alike", True), ("far", True), ("tiny", False),
                                       ("one triangle", False)])
def test_which_two_level_scenes_are_walked_wide(case, wide):
    """Inner trees wherever they lie, unless one has no wide nodes or is so small
    that rays reach it from beyond its origins' limit."""
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import InstancedBVH
    mesh = scenes.displaced_icosphere(3, seed=6)
    if case == "far":
        mesh = _far(mesh)
    if case == "tiny":
        mesh.vertices = (mesh.vertices * np.float32(1e-3)).astype(np.float32)
    if case == "one triangle":
        mesh = _soup(1, 1)
    inner = [_built(mesh), _built(scenes.heightfield(12, 10, 5, extent=3.0))]
    move = np.array([[0, 0, 0], [0, 0, 0], [3, 0.5, 1], [-2, 1, 2]], np.float32)
    if case == "far":
        move[[0, 2, 3]] -= np.float32(1e4)
    top = InstancedBVH(inner, np.array([0, 1, 0, 0], np.int32), move,
                       np.array([0, 1, 0, 0], np.int32))
    top.rebuild()
    assert _walks_wide(top) == wide
    top.close()
    for b in inner:
        b.close()
