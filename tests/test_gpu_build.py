"""GPU binned-SAH builder: valid trees, SAH cost within 2% of the
reference's exact-sweep DynBVH tree (costs recorded from the reference in
tests/golden/sah_costs.json: three small scenes and the benchmark scenes at
full size, 1.2M to 5.12M triangles), and traversal on the built tree
identical to the CPU restatement on the same (exported) tree."""
import json
import os
import sys

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

sys.path.insert(0, GOLDEN)


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _tree_of(bvh):
    from oracle.pyoracle import Tree
    from rfmanta_b200.treeio import parse_dynbvh_blob
    t = parse_dynbvh_blob(bvh.exportBlob())
    return Tree(t.bounds, t.child, t.children, t.axis, t.left_cheaper, t.ids)


SAH_COSTS = json.load(open(os.path.join(GOLDEN, "sah_costs.json")))


@pytest.mark.parametrize("name", sorted(SAH_COSTS))
def test_sah_cost_within_two_percent(name, restatement):
    import make_golden
    from rfmanta_b200.dynbvh import GpuDynBVH
    ref_cost = SAH_COSTS[name]
    mesh = make_golden.sah_scene_makers()[name]()
    bvh = GpuDynBVH()
    bvh.setGroup(mesh)
    bvh.rebuild()
    cost = bvh.sahCost()
    assert restatement.sah_cost(_tree_of(bvh)) == pytest.approx(cost, rel=1e-6)
    assert cost <= ref_cost * 1.02, (cost, ref_cost)
    # every triangle appears exactly once in the leaves
    t = _tree_of(bvh)
    assert np.array_equal(np.sort(t.ids), np.arange(mesh.n_tris))


@pytest.mark.parametrize("kind", [0, 1])
def test_traversal_on_built_tree(kind, restatement):
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH, RayBatch
    sc = scenes.small_frame_scene()
    bvh = GpuDynBVH(tri_kind=kind)
    bvh.setGroup(sc.mesh)
    bvh.rebuild()
    tree = _tree_of(bvh)
    lo, hi = sc.mesh.bounds()
    o, d, tm, any_mask = scenes.random_rays(200000, lo - 0.2, hi + 0.2, seed=31,
                                            anyhit_fraction=0.5)
    for anyhit in (False, True):
        sel = any_mask if anyhit else ~any_mask
        oo, dd, tt = o[:, sel].copy(), d[:, sel].copy(), tm[sel].copy()
        exp = restatement.trace(tree, sc.mesh, oo, dd, tt, anyhit=anyhit, tri_kind=kind)
        r = RayBatch(oo, dd, tt, flags=RayBatch.AnyHit if anyhit else 0)
        bvh.intersect(r)
        assert np.array_equal(r.wasHit(), exp["hit"] > 0)
        if not anyhit:
            assert np.array_equal(r.hitPrim, exp["prim"])
            assert np.array_equal(_bits(r.minT), _bits(exp["t"]))
    # the frame on the built tree equals the restatement's frame on that tree
    out = bvh.render_whitted(sc)
    exp = restatement.render_whitted(tree, sc, tri_kind=kind)
    assert out["shadow_rays"] == exp["shadow_rays"]
    assert np.array_equal(_bits(out["rgb"]), _bits(exp["rgb"]))


def test_degenerate_inputs():
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH, RayBatch
    # one triangle, two triangles, 1000 identical triangles (no usable split)
    tri = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
    for n in (1, 2, 1000):
        v = np.tile(tri, (n, 1))
        mesh = scenes.Mesh(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3),
                           np.zeros(n, np.uint32), np.ones((1, 3), np.float32))
        bvh = GpuDynBVH()
        bvh.setGroup(mesh)
        bvh.rebuild()
        t = _tree_of(bvh)
        assert np.array_equal(np.sort(t.ids), np.arange(n))
        r = RayBatch(np.array([[0.2], [0.2], [1.0]], np.float32),
                     np.array([[0.0], [0.0], [-1.0]], np.float32))
        bvh.intersect(r)
        assert r.hitPrim[0] >= 0 and abs(float(r.minT[0]) - 1.0) < 1e-6


def test_device_bytes_are_what_the_scene_holds():
    """rq_scene_info's figure against the device memory that making the scene took
    (the allocator's grain, 2 MB a block, aside)."""
    import torch
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH
    mesh = scenes.heightfield(700, 700, 3, extent=6.0)
    torch.cuda.synchronize()
    warm = GpuDynBVH()
    warm.setGroup(scenes.heightfield(8, 8, 3, extent=6.0))
    warm.rebuild()
    b = GpuDynBVH()
    b.setGroup(mesh)
    before = torch.cuda.mem_get_info()[0]
    b.rebuild()
    torch.cuda.synchronize()
    took = before - torch.cuda.mem_get_info()[0]
    said = b.info().device_bytes
    assert said > 100 << 20
    assert abs(took - said) < (32 << 20), (took, said)
    b.close()
    warm.close()
