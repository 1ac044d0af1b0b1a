"""The traversal's rounds (xtracer_b200/csrc/quad.cuh, wide.cuh) where they can go
wrong: primitives at equal distances, whose tie a box missed by a rounding would give
to another, and batches from one ray to more than there are lanes."""
import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu
FORMATS = (xtgpu.NODES_FP32, xtgpu.NODES_Q8, xtgpu.NODES_W8)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 12, 2.0 ** -12])
def test_equal_distances(scale):
    """A sheet of axis-aligned triangles on a dyadic grid, each three times over, seen from a thousandth of its
    size to its whole size away: child boxes that start at their node's origin, flat in one axis, and hits that
    tie.  Every format names the same primitive."""
    n = 24
    g = np.arange(n + 1) / 32.0
    x, y = np.meshgrid(g, g, indexing="ij")
    rng = np.random.default_rng(7)
    tris = []
    for axis in range(3):
        p = np.zeros((n + 1, n + 1, 3))
        p[..., axis], p[..., (axis + 1) % 3], p[..., (axis + 2) % 3] = 0.25, x, y
        a, b, c, e = p[:-1, :-1], p[1:, :-1], p[:-1, 1:], p[1:, 1:]
        tris += [np.stack([a, b, c], 2).reshape(-1, 3, 3), np.stack([b, e, c], 2).reshape(-1, 3, 3)]
    one = np.concatenate(tris)
    t = (np.concatenate([one, one[:, [1, 2, 0]], one[rng.permutation(len(one))]]) * scale).astype(np.float32)
    spec = scenes.hairball_scene(4, seed=1)
    spec.tris, spec.obj_count = t, np.array([len(t)], np.int32)
    at = t[rng.integers(0, len(t), 20000)].astype(np.float64).mean(1)
    d = rng.normal(size=(20000, 3))
    d[:2000] = np.eye(3)[rng.integers(0, 3, 2000)] * rng.choice([-1.0, 1.0], (2000, 1))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = at - d * scale * 2.0 ** rng.uniform(-10, 0, (20000, 1))
    o, d = o.astype(np.float32), d.astype(np.float32)
    want = None
    for leaf in (1, 3):
        sc = xtgpu.Scene(spec, node_formats=FORMATS, leaf_size=leaf)
        for fmt in FORMATS:
            h = sc.intersection(o, d, node_format=fmt)
            want = h if want is None else want
            np.testing.assert_array_equal(h.view(np.uint32), want.view(np.uint32))
        sc.close()
    assert np.isfinite(want["t"]).mean() > 0.9


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
