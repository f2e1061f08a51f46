"""Frame forms chosen by size: tiles of pixels or runs of samples, one pass or
several, wide or binary inner scenes - the same bits from each."""
import numpy as np
import pytest

from test_gpu_path import _bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp,sizes", [
    (1, [(8, 4), (40, 24), (9, 4), (8, 5), (1, 1)]), (4, [(4, 2), (20, 14), (21, 14), (20, 13)]),
    (16, [(2, 1), (18, 11), (19, 11)]), (9, [(8, 4), (7, 3)]), (64, [(6, 2)])])
def test_frame_samples_of_every_size(restatement, spp, sizes):
    """Widths and heights that tiles of 32 samples divide, and those they do not."""
    from conftest import golden_mesh, golden_tree, load_golden
    from test_gpu_render import _scene_from_golden
    from rfmanta_b200.dynbvh import GpuDynBVH
    g = load_golden("wald")
    sc = _scene_from_golden(g)
    b = GpuDynBVH()
    b.setGroup(golden_mesh(g))
    b.importTree(golden_tree(g))
    W = restatement.world(golden_tree(g), golden_mesh(g))
    sc.spp, sc.seed, sc.specular, sc.specpow = spp, 77, None, None
    for sc.xres, sc.yres in sizes:
        out = b.render_frame(sc, sc.mesh.materials)
        exp = restatement.render_frame(W, sc, sc.mesh.materials)
        assert out["shadow_rays"] == exp["shadow_rays"]
        assert np.array_equal(_bits(out["rgb"]), _bits(exp["rgb"]))
    b.close()


@pytest.mark.parametrize("case", ["alike", "far", "tiny", "one triangle"])
def test_two_level_walks_agree(restatement, case):
    """Inner scenes far from their own origin, far smaller than the whole, or
    without wide nodes (then all take the binary walk)."""
    import torch
    from oracle.pyoracle import Tree
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH, InstancedBVH
    from rfmanta_b200.scenes import Mesh
    from rfmanta_b200.treeio import parse_dynbvh_blob
    from test_gpu_instance import _trace
    meshes = [scenes.displaced_icosphere(3, seed=6), scenes.heightfield(12, 10, 5, extent=3.0)]
    if case == "far":
        meshes[0].vertices = (meshes[0].vertices + np.float32(500.0)).astype(np.float32)
    if case == "tiny":
        meshes[0].vertices = (meshes[0].vertices * np.float32(1e-3)).astype(np.float32)
    if case == "one triangle":
        meshes[0] = Mesh(np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]], np.float32),
                         np.array([[0, 1, 2]], np.uint32), np.zeros(1, np.uint32),
                         np.full((1, 3), 0.5, np.float32))
    inner = []
    for m in meshes:
        b = GpuDynBVH()
        b.setGroup(m)
        b.rebuild()
        inner.append(b)
    which = np.array([0, 1, 0, 0, 1], np.int32)
    move = np.array([[0, 0, 0], [0, 0, 0], [3, 0.5, 1], [-2, 1, 2], [1, 2, -3]], np.float32)
    if case == "far":
        move[which == 0] -= np.float32(500.0)
    kind = np.array([0, 1, 0, 0, 0], np.int32)  # one nested in place
    top = InstancedBVH(inner, which, move, kind)
    top.rebuild()

    def exported(b, n):
        f = parse_dynbvh_blob(b.exportBlob(), n)
        return Tree(f.bounds, f.child, f.children, f.axis, f.left_cheaper, f.ids)
    W = restatement.world(exported(top, top.n_instances),
                          inner=[(exported(b, m.n_tris), m) for b, m in zip(inner, meshes)],
                          inst_scene=which, translation=move, kind=kind)
    rng = np.random.default_rng(8)
    n = 4000
    org = rng.uniform(-6, 6, (3, n)).astype(np.float32)
    aim = (move[rng.integers(0, 5, n)].T + rng.normal(scale=0.4, size=(3, n))).astype(np.float32)
    if case == "far":
        aim += np.float32(500.0) * (rng.random(n) < 0.5)
    if case == "tiny":
        aim[:, ::2] = (move[rng.choice([0, 2, 3], (n + 1) // 2)].T +
                       rng.normal(scale=1e-3, size=(3, (n + 1) // 2)))
    d = (aim - org).astype(np.float32)
    d[0, ::50] = 0.0          # no finite inverse
    d[1, 1::50] *= 1e-6       # too steep for the wide walk
    org[:, 2::50] *= 1000.0   # too far for it
    for anyhit in (False, True):
        tmax = np.full(n, 1e19, np.float32)
        got = _trace(top, org, d, tmax, anyhit)
        exp = restatement.trace_world(W, org, d, tmax, anyhit)
        assert np.array_equal(got["prim"], exp["prim"])
        if not anyhit:
            assert np.array_equal(got["inst"], exp["inst"])
            for k in ("t", "u", "v"):
                assert np.array_equal(_bits(got[k]), _bits(exp[k])), k
    top.close()


def test_recorded_path_frames_and_larger_ones():
    """A path frame recorded in a CUDA graph replays correctly after larger
    frames replaced the scene's buffers, and a frame larger than the buffers can
    be recorded (in passes that fit them)."""
    import torch
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH
    sc = scenes.tiny_path_scene()
    b = GpuDynBVH()
    b.setGroup(sc.mesh)
    b.rebuild()

    def record(sc):
        p = b.path_params(sc)
        rgb = torch.zeros(sc.xres * sc.yres * 3, device="cuda")
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            b.render_path_device(p, rgb.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
        return g, rgb, p

    big = scenes.tiny_path_scene(61, 47, 9)
    small = b.render_path(sc)["rgb"]
    recorded = [(sc, record(sc)), (big, record(big))]
    frames = {sc.xres: small, big.xres: b.render_path(big)["rgb"]}
    b.render_path(scenes.tiny_path_scene(150, 100, 16))
    junk = torch.full((1 << 24,), float("nan"), device="cuda")
    for s, (g, rgb, p) in recorded:
        rgb.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(_bits(rgb.cpu().numpy().reshape(-1, 3)), _bits(frames[s.xres]))
    del recorded, junk
    b.close()
