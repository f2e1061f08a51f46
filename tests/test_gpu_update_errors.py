"""Updates that fail part way: the call's error, the scene afterwards, and
everything else that uses the device or the scene."""
import numpy as np
import pytest

LIMIT = 512  # traversal stack entries: a tree of this depth is refused


def _deep(depth, bottom=8):
    """A chain of `depth` records over triangles that shrink by 0.95 a level
    (rotations do not pay), ending in a leaf of `bottom` small, separate ones
    that an update splits into a chain of its own, three levels deep."""
    from oracle.pyoracle import Tree
    from rfmanta_b200.scenes import Mesh
    n = depth + bottom
    size = (0.95 ** np.minimum(np.arange(n), depth)).astype(np.float32)
    base = np.array([[0, 0, 0], [1, 0, 0], [0, 1, .3]], np.float32)
    v = (base[None] * size[:, None, None]).astype(np.float32)
    e = size[depth - 1]
    for j in range(bottom):
        v[depth + j] = base * (e * 1e-3) + np.array([e * .9 * j / bottom, 0, 0], np.float32)
    lo, hi = v.min(1), v.max(1)
    nodes = 2 * depth + 1
    bounds = np.zeros((nodes, 6), np.float32)
    child = np.zeros(nodes, np.int32)
    children = np.zeros(nodes, np.int32)
    for k in range(depth):  # node 2k+1: triangle k; node 2k+2: the rest
        child[2 * k] = 2 * k + 1
        child[2 * k + 1], children[2 * k + 1] = k, 1
        bounds[2 * k + 1] = np.concatenate([lo[k], hi[k]])
    child[nodes - 1], children[nodes - 1] = depth, bottom
    for k in range(depth + 1):
        bounds[2 * k] = np.concatenate([lo[k:].min(0), hi[k:].max(0)])
    mesh = Mesh(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(n, 3),
                np.zeros(n, np.uint32), np.full((1, 3), 0.5, np.float32))
    return mesh, Tree(bounds, child, children, (np.arange(nodes) % 3).astype(np.uint8),
                      (np.arange(nodes) % 2).astype(np.uint8), np.arange(n, dtype=np.int32))


def _depth(t):
    deepest, todo = 0, [(0, 0)]
    while todo:
        i, d = todo.pop()
        deepest = max(deepest, d)
        if t.children[i] == 0:
            todo += [(int(t.child[i]), d + 1), (int(t.child[i]) + 1, d + 1)]
    return deepest


@pytest.mark.parametrize("depth,after", [(LIMIT - 4, LIMIT - 1), (LIMIT - 2, LIMIT + 1)])
def test_the_update_deepens_the_chain(restatement, depth, after):
    """The trees of the device test below cross the limit by the update, and
    only the second one does (on the CPU restatement)."""
    from oracle.pyoracle import DynTree
    mesh, tree = _deep(depth)
    d = DynTree(tree, mesh.n_tris, next_free=tree.children.shape[0])
    restatement.tree_costs(d)
    restatement.tree_update(d, mesh.vertices, mesh.indices, rotate=True)
    assert (_depth(tree), _depth(d.tree())) == (depth, after)


def _sphere():
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH
    b = GpuDynBVH()
    b.setGroup(scenes.displaced_icosphere(3, seed=4))
    b.rebuild()
    return b


def _hits(bvh):
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import RayBatch
    o, d, tm, _ = scenes.random_rays(4096, np.full(3, -2.0), np.full(3, 2.0), seed=3,
                                     anyhit_fraction=0.0)
    r = RayBatch(o, d, np.full(o.shape[1], 1e19, np.float32))
    bvh.intersect(r)
    return r


@pytest.mark.gpu
def test_an_update_that_grows_too_deep_is_an_error_and_no_more():
    from rfmanta_b200._lib import RQ_ERR_CAPACITY, RQ_ERR_STATE, RQError
    from rfmanta_b200.dynbvh import GpuDynBVH
    other = _sphere()
    want = _hits(other)
    mesh, tree = _deep(LIMIT - 4)
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.importTree(tree)
    b.update(rotate=True)
    assert b.info().depth == LIMIT - 1
    b.close()
    mesh, tree = _deep(LIMIT - 2)
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.importTree(tree)
    with pytest.raises(RQError) as e:
        b.update(rotate=True)
    assert e.value.code == RQ_ERR_CAPACITY
    with pytest.raises(RQError) as e:  # the tree is gone, and says so
        _hits(b)
    assert e.value.code == RQ_ERR_STATE
    got = _hits(other)
    assert np.array_equal(got.hitPrim, want.hitPrim) and np.array_equal(got.minT, want.minT)
    b.rebuild()  # and can be made again
    assert _hits(b).hitPrim.shape == want.hitPrim.shape
    b.close()
    other.close()


@pytest.mark.gpu
def test_an_update_out_of_memory_leaves_the_scene_as_it_was():
    """Every device allocation of the first rotating update fails in turn:
    the record buffers have moved by then, and the scene and a plan made
    before it give the answers they gave."""
    import torch
    from rfmanta_b200 import _lib, scenes
    from rfmanta_b200.batch import BatchedQueries, QueryBatch
    b = _sphere()
    o, d, _, _ = scenes.random_rays(4096, np.full(3, -2.0), np.full(3, 2.0), seed=5,
                                    anyhit_fraction=0.0)
    q = QueryBatch(0, *(torch.from_numpy(x).cuda() for x in (o, d)),
                   torch.full((o.shape[1],), 1e19, device="cuda"))
    plan = BatchedQueries([b], [q])

    def answers():
        plan.launch()
        torch.cuda.synchronize()
        r = _hits(b)
        return [plan.t[0].cpu().numpy(), plan.prim[0].cpu().numpy(), r.minT, r.hitPrim]

    want = answers()
    failed = 0
    for nth in range(1, 64):
        _lib.check(_lib.lib.rq_fail_allocation(nth))
        try:
            b.update(rotate=True)
        except _lib.RQError as e:
            assert e.code == _lib.RQ_ERR_OOM
            failed += 1
        else:
            break
        finally:
            _lib.lib.rq_fail_allocation(0)
        for got, w in zip(answers(), want):
            assert np.array_equal(got, w)
    assert 10 < failed < 63
    got = answers()  # (the update moved no vertex: the same hits from the rotated tree)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[2], want[2])
    plan.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nth", [1, 2, 3])
def test_a_plan_refuses_a_scene_that_lost_its_tree(nth):
    """An import out of memory has freed the old tree, which the plan's table
    still points at."""
    import torch
    from rfmanta_b200 import _lib
    from rfmanta_b200.batch import BatchedQueries, QueryBatch
    b = _sphere()
    blob = b.exportBlob()
    n = 64
    q = QueryBatch(0, torch.zeros(3, n, device="cuda"), torch.ones(3, n, device="cuda"),
                   torch.ones(n, device="cuda"))
    plan = BatchedQueries([b], [q])
    plan.launch()
    torch.cuda.synchronize()
    _lib.check(_lib.lib.rq_fail_allocation(nth))
    try:
        with pytest.raises(_lib.RQError) as e:
            b.importBlob(blob)
        assert e.value.code == _lib.RQ_ERR_OOM
    finally:
        _lib.lib.rq_fail_allocation(0)
    with pytest.raises(_lib.RQError) as e:
        plan.launch()
    assert e.value.code == _lib.RQ_ERR_STATE
    b.importBlob(blob)
    plan.launch()
    torch.cuda.synchronize()
    plan.close()
    b.close()


@pytest.mark.gpu
def test_a_refused_call_is_not_the_next_ones_error():
    """Queries and frames of a tree whose stack does not fit are refused by the
    runtime, on the host; the scene takes its next tree all the same."""
    from rfmanta_b200 import _lib, scenes
    from rfmanta_b200.dynbvh import GpuDynBVH
    mesh, tree = _deep(LIMIT - 4)
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.rebuild()
    blob = b.exportBlob()
    want = _hits(b)
    sc = scenes.tiny_frame_scene()
    sc.mesh = mesh
    for refused in (lambda: _hits(b), lambda: b.render_whitted(sc)):
        b.importTree(tree)
        with pytest.raises(_lib.RQError):
            refused()
        b.importBlob(blob)
        b.update(rotate=True)
        b.importBlob(blob)
        assert np.array_equal(_hits(b).minT, want.minT)
    b.close()


@pytest.mark.gpu
def test_a_plan_waits_for_a_tree_it_can_take():
    """A tree too deep for the plan's stack is an error at every launch (the old
    graph would read the freed tree), and the plan runs again with the next one."""
    import torch
    from rfmanta_b200 import _lib, scenes
    from rfmanta_b200.batch import BatchedQueries, QueryBatch
    from rfmanta_b200.dynbvh import GpuDynBVH
    mesh, tree = _deep(LIMIT - 4)
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.rebuild()
    blob = b.exportBlob()
    o, d, _, _ = scenes.random_rays(4096, np.full(3, -1.0), np.full(3, 1.0), seed=7,
                                    anyhit_fraction=0.0)
    q = QueryBatch(0, *(torch.from_numpy(x).cuda() for x in (o, d)),
                   torch.full((o.shape[1],), 1e19, device="cuda"))
    plan = BatchedQueries([b], [q])
    plan.launch()
    torch.cuda.synchronize()
    want = [plan.t[0].cpu().numpy(), plan.prim[0].cpu().numpy()]
    b.importTree(tree)
    for _ in range(2):
        with pytest.raises(_lib.RQError) as e:
            plan.launch()
        assert e.value.code == _lib.RQ_ERR_CAPACITY
    b.importBlob(blob)
    plan.t[0].zero_()
    plan.launch()
    torch.cuda.synchronize()
    for got, w in zip((plan.t[0].cpu().numpy(), plan.prim[0].cpu().numpy()), want):
        assert np.array_equal(got, w)
    plan.close()
    b.close()
