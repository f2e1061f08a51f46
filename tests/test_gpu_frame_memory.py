"""Device memory of Whitted, supersampled and path frames: what a frame after a failed
allocation does, and what recorded frames hold."""
import numpy as np
import pytest

from test_gpu_path import _bits

pytestmark = pytest.mark.gpu


def _built(mesh):
    from rfmanta_b200.dynbvh import GpuDynBVH
    b = GpuDynBVH()
    b.setGroup(mesh)
    b.rebuild()
    return b


def _whitted(x=40, y=32):
    from rfmanta_b200 import scenes
    sc = scenes.tiny_frame_scene()
    sc.xres, sc.yres = x, y
    return sc


def _phong(x=40, y=32):
    sc = _whitted(x, y)
    k = sc.mesh.materials.shape[0]
    sc.spp, sc.seed = 4, 9
    sc.specular = np.full((k, 3), 0.4, np.float32)
    sc.specpow = np.full(k, 12, np.int32)
    sc.reflectivity = np.full(k, 0.3, np.float32)
    sc.max_depth = 3
    return sc


def _path(x=40, y=32):
    from rfmanta_b200 import scenes
    return scenes.tiny_path_scene(x, y, 4)


KINDS = {"whitted": (_whitted, lambda b, sc: b.render_whitted(sc)["rgb"]),
         "supersampled": (_phong, lambda b, sc: b.render_frame(sc, sc.mesh.materials)["rgb"]),
         "path": (_path, lambda b, sc: b.render_path(sc)["rgb"])}


def _other_materials(sc, k):
    sc.mesh.materials = (sc.mesh.materials * np.float32(0.9 - 0.2 * k)).astype(np.float32)
    if hasattr(sc, "specular"):
        sc.specular = (sc.specular * np.float32(0.5)).astype(np.float32)
        sc.specpow = sc.specpow + 1
        sc.reflectivity = (sc.reflectivity * np.float32(0.5)).astype(np.float32)
    return sc


@pytest.mark.parametrize("kind", list(KINDS))
def test_frames_after_failed_allocations(kind):
    """Each allocation of a frame larger than the one before, with other materials,
    fails in turn; the first frame's scene, size and materials then give the first
    image again."""
    from rfmanta_b200 import _lib
    make, render = KINDS[kind]
    sc = make()
    b = _built(sc.mesh)
    own = sc.mesh.materials.copy()
    want = render(b, sc)
    failed = 0
    for nth in range(1, 32):
        big = _other_materials(make(80 + nth, 64), 1)
        _lib.check(_lib.lib.rq_fail_allocation(nth))
        try:
            render(b, big)
        except _lib.RQError as e:
            assert e.code == _lib.RQ_ERR_OOM
            failed += 1
        finally:
            left = _lib.lib.rq_fail_allocation(0)
            assert left == 0
        sc = make()
        assert np.array_equal(sc.mesh.materials, own)
        assert np.array_equal(_bits(render(b, sc)), _bits(want))
    assert failed >= 2
    b.close()


@pytest.mark.parametrize("kind", list(KINDS))
def test_recorded_frames_keep_what_they_hold(kind):
    """A frame recorded into a CUDA graph replays after frames with other tables and
    larger ones."""
    import torch
    make, render = KINDS[kind]
    sc = make()
    b = _built(sc.mesh)
    want = render(b, sc)
    n = sc.xres * sc.yres
    rgb = torch.zeros(3 * n, device="cuda")
    t = torch.zeros(n, device="cuda")
    prim = torch.zeros(n, dtype=torch.int32, device="cuda")
    p = {"whitted": lambda: b.whitted_params(sc),
         "supersampled": lambda: b.frame_params(sc, sc.mesh.materials),
         "path": lambda: b.path_params(sc)}[kind]()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        st = torch.cuda.current_stream().cuda_stream
        if kind == "whitted":
            b.render_whitted_device(p, rgb.data_ptr(), t.data_ptr(), prim.data_ptr(), 0, st)
        elif kind == "supersampled":
            b.render_frame_device(p, rgb.data_ptr(), 0, st)
        else:
            b.render_path_device(p, rgb.data_ptr(), 0, st)
    for k in range(3):
        render(b, _other_materials(make(60 + 40 * k, 48 + 40 * k), k))
    junk = [torch.full((1 << 10,), 7.0, device="cuda") for _ in range(64)]
    junk.append(torch.full((1 << 22,), 7.0, device="cuda"))
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(_bits(rgb.cpu().numpy().reshape(-1, 3)), _bits(want))
    assert np.array_equal(_bits(render(b, make())), _bits(want))
    del g, junk
    b.close()
