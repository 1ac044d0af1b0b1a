"""xtgpu_release_memory: what closed scenes leave goes back to the driver, and open ones are not touched."""
import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu


def test_release_memory():
    import torch
    keep = xtgpu.Scene(scenes.hairball_scene(5000, seed=1), node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_W8), leaf_size=1)
    want = keep.render(xtgpu.AO, 64, 48, 2, seed=3, node_format=xtgpu.NODES_W8)[0]
    xtgpu.release_memory()
    before = torch.cuda.mem_get_info()[0]
    sc = xtgpu.Scene(scenes.terrain_scene(300_000, seed=1), leaf_size=1)
    held = sc.device_bytes()
    sc.close()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept >= held // 2   # the blocks are still the library's
    assert xtgpu.release_memory() >= held
    assert before - torch.cuda.mem_get_info()[0] <= 4 << 20
    np.testing.assert_array_equal(keep.render(xtgpu.AO, 64, 48, 2, seed=3, node_format=xtgpu.NODES_W8)[0], want)
    keep.close()
