"""Device memory of path frames: what recorded frames hold, and what a frame does
when memory is short."""
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
