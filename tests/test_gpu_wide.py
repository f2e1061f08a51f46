"""The wide walk (rq_wide.cuh) against the binary walk it replaces, bit for bit.

A batch plan with register stack entries runs the binary walk over the node
records, the default plan and rq_trace the wide one; every form of ray and
tree the wide rule accepts or refuses must give the same t, triangle id, u and
v from both.  No tolerance: the two walks make the same accepting tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _grid(n, y=0.0, scale=1.0, offset=(0.0, 0.0, 0.0)):
    from rfmanta_b200 import scenes
    m = scenes.quad_grid(n, n, -1.0, 1.0, -1.0, 1.0, y=y)
    m.vertices = (m.vertices * np.float32(scale) + np.asarray(offset, np.float32)).astype(np.float32)
    return m


def _soup(n, seed, spread=1.0):
    from rfmanta_b200.scenes import Mesh
    rng = np.random.default_rng(seed)
    c = rng.uniform(-spread, spread, (n, 1, 3))
    v = (c + rng.normal(scale=0.2, size=(n, 3, 3))).astype(np.float32).reshape(-1, 3)
    return Mesh(v, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), np.zeros(n, np.uint32),
                np.full((1, 3), 0.5, np.float32))


def _doubled(m):
    """Every triangle twice: equal distances everywhere."""
    from rfmanta_b200.scenes import Mesh
    return Mesh(m.vertices, np.concatenate([m.indices, m.indices]),
                np.concatenate([m.face_material] * 2), m.materials)


def _meshes():
    from rfmanta_b200 import scenes
    yield "one", _soup(1, 1)
    yield "two", _soup(2, 2)
    yield "three", _soup(3, 3)
    yield "five", _soup(5, 5)
    yield "soup", _soup(700, 7)
    yield "flat", _grid(17)
    yield "small far away", _grid(9, scale=1e-3, offset=(100.0, -40.0, 7.0))
    yield "doubled", _doubled(scenes.displaced_icosphere(2, seed=3))
    yield "sphere", scenes.displaced_icosphere(4, seed=4)
    yield "heightfield", scenes.heightfield(48, 40, 5, extent=4.0)


MESHES = ["one", "two", "three", "five", "soup", "flat", "small far away", "doubled", "sphere",
          "heightfield"]


def _rays(mesh, seed):
    """Ordinary rays and those at the edges of the wide rule: directions with
    zero, tiny and huge components, origins on vertex coordinates and far
    outside, infinite, zero, negative and NaN upper bounds."""
    rng = np.random.default_rng(seed)
    lo, hi = (x.astype(np.float64) for x in mesh.bounds())
    ext = max(float((hi - lo).max()), 1e-6)
    v = mesh.vertices
    parts = []

    def add(o, d, t):
        n = o.shape[0]
        parts.append((o.astype(np.float32), d.astype(np.float32),
                      np.broadcast_to(np.asarray(t, np.float32), (n,))))

    def unit(n):
        d = rng.normal(size=(n, 3))
        return d / np.linalg.norm(d, axis=1, keepdims=True)

    n = 1500
    inside = lo - 0.3 * ext + (hi - lo + 0.6 * ext) * rng.random((n, 3))
    target = v[rng.integers(0, v.shape[0], n)] + rng.normal(scale=0.05 * ext, size=(n, 3))
    add(inside, unit(n), 1e19)
    add(inside, unit(n), rng.uniform(0, 2 * ext, n))
    add(inside, target - inside, 1.0)              # unnormalised, ends at the target
    add(inside, (target - inside) * 1e-7, np.inf)
    add(inside, (target - inside) * 1e7, 1e19)
    for far in (3.0, 10.0, 40.0, 1e4):             # origins far outside
        o = target + unit(n) * far * max(ext, float(np.abs(v).max()))
        add(o, target - o, np.inf)
    for k in range(3):                             # along an axis, through vertices too
        d = np.zeros((n, 3))
        d[:, k] = rng.choice([-1.0, 1.0], n)
        o = v[rng.integers(0, v.shape[0], n)].astype(np.float64)
        o[: n // 2] += rng.normal(scale=0.01 * ext, size=(n // 2, 3))
        o -= d * ext
        add(o, d, 1e19)
        d2 = unit(n)
        d2[:, k] = rng.choice([0.0, -0.0, 1e-30, -1e-6, 1e-4, 3e-4], n)  # in or near a plane
        o2 = v[rng.integers(0, v.shape[0], n)].astype(np.float64)
        add(o2 - d2 * ext, d2, 1e19)
    edge = v[rng.integers(0, v.shape[0], n)]       # exactly at vertices
    add(inside, edge - inside, 1e19)
    add(inside[:200], unit(200), 0.0)
    add(inside[:200], unit(200), -1.0)
    add(inside[:200], unit(200), np.nan)
    bad = unit(64)
    bad[:32, 0] = np.nan
    bad[32:] = 0.0
    add(inside[:64], bad, 1e19)
    bo = inside[:64].copy()
    bo[:, 1] = np.inf
    add(bo, unit(64), 1e19)
    o, d, t = (np.concatenate(x) for x in zip(*parts))
    return np.ascontiguousarray(o.T), np.ascontiguousarray(d.T), np.ascontiguousarray(t)


def _compare(bvh, mesh, seed):
    import torch
    from rfmanta_b200.batch import BatchedQueries, QueryBatch
    from rfmanta_b200.dynbvh import RayBatch
    o, d, t = _rays(mesh, seed)
    dev = [torch.from_numpy(x).cuda() for x in (o, d, t)]
    for anyhit in (False, True):
        plans = [BatchedQueries([bvh], [QueryBatch(0, *dev, anyhit, want_uv=True)], cfg)
                 for cfg in (None, dict(reg_stack=1))]
        for p in plans:
            p.launch()
        torch.cuda.synchronize()
        wide, binary = ([x[0].cpu().numpy() for x in (p.t, p.prim, p.u, p.v)] for p in plans)
        r = RayBatch(o, d, t, flags=RayBatch.AnyHit if anyhit else 0)
        bvh.intersect(r)
        k = 777  # a packet-sized call: one thread per ray
        q = RayBatch(o[:, :k], d[:, :k], t[:k], flags=RayBatch.AnyHit if anyhit else 0)
        bvh.intersect(q)
        for a in (wide, [r.minT, r.hitPrim, r.u, r.v]):
            assert np.array_equal(a[1], binary[1])
            for i in (0, 2, 3):
                assert np.array_equal(_bits(a[i]), _bits(binary[i]))
        assert np.array_equal(q.hitPrim, binary[1][:k])
        assert np.array_equal(_bits(q.minT), _bits(binary[0][:k]))
        for p in plans:
            p.close()


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("name", MESHES)
def test_wide_walk_is_the_binary_walk(name, kind):
    from rfmanta_b200.dynbvh import GpuDynBVH
    mesh = dict(_meshes())[name]
    b = GpuDynBVH(tri_kind=kind)
    b.setGroup(mesh)
    b.rebuild()
    _compare(b, mesh, seed=11)
    if mesh.n_tris > 1:  # the wide nodes follow the tree's updates
        for k, rotate in enumerate((True, False, True)):
            rng = np.random.default_rng(20 + k)
            mesh.vertices = (mesh.vertices + rng.normal(
                scale=0.02 * float(np.ptp(mesh.vertices)), size=mesh.vertices.shape)
            ).astype(np.float32)
            b.update(rotate=rotate)
            _compare(b, mesh, seed=30 + k)
    b.close()


def test_trees_the_wide_walk_refuses():
    """Boxes that are not nested, and a tree deeper than the wide walk takes:
    both are traced as before, over the node records."""
    from rfmanta_b200.dynbvh import GpuDynBVH
    from rfmanta_b200.treeio import TreeFields, parse_dynbvh_blob
    mesh = _soup(300, 9)
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.rebuild()
    t = parse_dynbvh_blob(b.exportBlob(), mesh.n_tris)
    inner = np.nonzero((t.children == 0) & (np.arange(t.children.shape[0]) > 0))[0]
    for i in inner[:20]:  # shrink some inner boxes below their children's
        c = (t.bounds[i, :3] + t.bounds[i, 3:]) / 2
        t.bounds[i] = np.concatenate([c, c]) + 0.4 * (t.bounds[i] - np.concatenate([c, c]))
    b.importTree(t)
    _compare(b, mesh, seed=41)
    b.close()
    n = 100  # a chain: node 2k+1 a leaf, node 2k+2 the rest
    mesh = _soup(n, 10, spread=2.0)
    tri = mesh.vertices.reshape(n, 3, 3)
    lo, hi = tri.min(1), tri.max(1)
    nodes = 2 * n - 1
    bounds = np.zeros((nodes, 6), np.float32)
    child = np.zeros(nodes, np.int32)
    children = np.zeros(nodes, np.int32)
    for k in range(n - 1):
        top = 0 if k == 0 else 2 * k
        child[top] = 2 * k + 1
        child[2 * k + 1], children[2 * k + 1] = k, 1
        bounds[2 * k + 1] = np.concatenate([lo[k], hi[k]])
    child[nodes - 1], children[nodes - 1] = n - 1, 1
    for k in range(n):
        i = 0 if k == 0 else 2 * k
        bounds[i] = np.concatenate([lo[k:].min(0), hi[k:].max(0)])
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.importTree(TreeFields(bounds, child, children, (np.arange(nodes) % 3).astype(np.uint8),
                            (np.arange(nodes) % 2).astype(np.uint8),
                            np.arange(n, dtype=np.int32)))
    assert b.info().depth > 64
    _compare(b, mesh, seed=42)
    b.close()
