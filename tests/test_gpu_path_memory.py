"""Device memory of path frames: what recorded frames hold, and what a frame does
when memory is short."""
import dataclasses

import numpy as np
import pytest

from test_gpu_path import _bits

pytestmark = pytest.mark.gpu


@pytest.fixture
def tiny():
    from rfmanta_b200 import scenes
    from rfmanta_b200.dynbvh import GpuDynBVH
    sc = scenes.tiny_path_scene()
    b = GpuDynBVH()
    b.setGroup(sc.mesh)
    b.rebuild()
    yield sc, b
    b.close()


def test_recorded_frame_keeps_its_materials(tiny):
    """Frames with other materials come between the recording and the replay."""
    import torch
    sc, b = tiny
    own = sc.mesh.materials.copy()
    want = b.render_path(sc)["rgb"]
    p = b.path_params(sc)
    rgb = torch.zeros(sc.xres * sc.yres * 3, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.render_path_device(p, rgb.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    for k in range(3):
        sc.mesh.materials = (own * np.float32(0.2 + 0.3 * k)).astype(np.float32)
        other = b.render_path(sc)["rgb"]
        assert not np.array_equal(other, want)
    junk = [torch.full((1 << 10,), 7.0, device="cuda") for _ in range(64)]
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(_bits(rgb.cpu().numpy().reshape(-1, 3)), _bits(want))
    sc.mesh.materials = own
    assert np.array_equal(_bits(b.render_path(sc)["rgb"]), _bits(want))
    del g, junk


def test_frames_when_memory_is_short(tiny):
    """The pass that does not fit is halved, and the next frame of that size
    allocates nothing; an explicit pass is one allocation and its error; an
    explicit larger pass takes the place of the buffers there."""
    from rfmanta_b200 import _lib, scenes
    _, b = tiny
    sc = scenes.tiny_path_scene(512, 512, 9)  # 2.36 Mi paths
    fail = _lib.lib.rq_fail_allocation
    want = b.render_path(scenes.tiny_path_scene(512, 512, 9), chunk_paths=1 << 18)["rgb"]
    try:
        fail(1)
        with pytest.raises(_lib.RQError) as e:  # the scene's first frame has nothing to give up
            _fresh(sc).render_path(sc, chunk_paths=1 << 20)
        assert e.value.code == _lib.RQ_ERR_OOM
        c = _fresh(sc)
        fail(1)
        assert np.array_equal(_bits(c.render_path(sc)["rgb"]), _bits(want))
        fail(1)  # stays armed: no allocation is left to fail
        assert np.array_equal(_bits(c.render_path(sc)["rgb"]), _bits(want))
        assert np.array_equal(_bits(c.render_path(scenes.tiny_path_scene(512, 512, 9))["rgb"]),
                              _bits(want))
        # (armed still) the larger pass fails once, the old buffers go, it fits
        assert np.array_equal(_bits(c.render_path(sc, chunk_paths=1 << 22)["rgb"]), _bits(want))
        c.close()
    finally:
        fail(0)


def _fresh(sc):
    from rfmanta_b200.dynbvh import GpuDynBVH
    b = GpuDynBVH()
    b.setGroup(sc.mesh)
    b.rebuild()
    return b


def test_debug_dumps_are_one_pass_of_at_most_4_mi_paths(tiny):
    import torch
    from rfmanta_b200 import _lib, scenes
    _, b = tiny
    for x, taken in ((1024, True), (1025, False)):
        sc = dataclasses.replace(scenes.tiny_path_scene(x, 1024, 4), max_depth=1)
        n = x * 1024 * 4
        prim = torch.zeros(n, dtype=torch.int32, device="cuda")
        od = torch.zeros(6 * n, device="cuda")
        b.set_path_debug(prim.data_ptr(), od.data_ptr(), od[3 * n:].data_ptr(), n)
        if taken:
            b.render_path(sc)
        else:
            with pytest.raises(_lib.RQError) as e:
                b.render_path(sc)
            assert e.value.code == _lib.RQ_ERR_ARG
            b.render_path(sc, chunk_paths=n)  # one pass by the caller's choice
        b.set_path_debug(0, 0, 0, 0)


def test_a_dump_after_a_larger_frame(tiny):
    """The dump's rows are as long as the caller says, whatever the buffers hold."""
    import torch
    from rfmanta_b200 import scenes
    sc, b = tiny
    n, D = sc.xres * sc.yres * sc.spp, sc.max_depth

    def dump(cap):
        pad = 1 << 16  # behind each array: must stay as it is
        prim = torch.full((D * cap + pad,), -2, dtype=torch.int32, device="cuda")
        od = [torch.full((3 * D * cap + pad,), -2.0, device="cuda") for _ in range(2)]
        b.set_path_debug(prim.data_ptr(), od[0].data_ptr(), od[1].data_ptr(), cap)
        b.render_path(sc)
        b.set_path_debug(0, 0, 0, 0)
        assert all(bool((x[-pad:] == -2).all()) for x in (prim, *od))
        return [x[:-pad].cpu().numpy().reshape(-1, cap)[:, :n] for x in (prim, *od)]

    want = dump(n)
    b.render_path(scenes.tiny_path_scene(150, 100, 16))
    for cap in (n, n + 5):
        for got, w in zip(dump(cap), want):
            assert np.array_equal(got, w)
