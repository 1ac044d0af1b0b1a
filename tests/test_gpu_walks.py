"""The traversal's rounds (xtracer_b200/csrc/quad.cuh, wide.cuh) where they can go
wrong, batches from one ray to more than there are lanes, and the bounce shading
(render.cu, k_shade), which gathers the hits of 32-path chunks."""
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


@pytest.mark.parametrize("kind", [xtgpu.PATHTRACER, xtgpu.AO])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (31, 1, 1), (1, 33, 1), (63, 5, 3), (301, 17, 64)])
def test_gathered_hits(kind, w, h, spp):
    """A rectangle's pixels are those of the whole frame, whose waves put other paths beside theirs: fewer bounce
    rays than a warp, part of a chunk, and several chunks a warp, on one material and on diffuse and specular ones."""
    for spec in (scenes.spheres_scene(40, seed=3), scenes.phong_scene()):
        sc = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_FP32,), leaf_size=1)
        whole = sc.render(kind, 403, 307, spp, 5, 100.0, 11)[0]
        part = sc.render(kind, 403, 307, spp, 5, 100.0, 11, rect=(51, 143, 51 + w, 143 + h))[0]
        sc.close()
        np.testing.assert_array_equal(part.view(np.uint32), whole[143:143 + h, 51:51 + w].view(np.uint32))
