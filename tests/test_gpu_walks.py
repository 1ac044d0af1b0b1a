"""The traversal's rounds (xtracer_b200/csrc/quad.cuh, wide.cuh) where they can go
wrong: batches from one ray to more than there are lanes."""
import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu
FORMATS = (xtgpu.NODES_FP32, xtgpu.NODES_Q8, xtgpu.NODES_W8)


@pytest.mark.parametrize("n", [1, 2, 33, 4735, 4737, 9473, 18943, 18945])
def test_small_batches(n):
    """A warp that has few rays leaves lanes idle (one warp of 4736 to 18944 rays takes one to four): the hits are
    those of a large batch."""
    sc = xtgpu.Scene(scenes.hairball_scene(20000, seed=5), node_formats=FORMATS, leaf_size=1)
    rng = np.random.default_rng(3)
    o = rng.normal(size=(30000, 3)).astype(np.float32)
    d = rng.normal(size=(30000, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    for fmt in FORMATS:
        whole = sc.intersection(o, d, node_format=fmt)
        part = sc.intersection(o[:n], d[:n], node_format=fmt)
        np.testing.assert_array_equal(part.view(np.uint32), whole[:n].view(np.uint32))
    sc.close()
