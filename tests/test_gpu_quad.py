"""FP32 and Q8 trees of four-child nodes (xtracer_b200/csrc/quad.cuh) where they
can go wrong: one primitive to a few, so that the root is a leaf, a node with
empty slots or a node over nodes; every leaf size, node order and hierarchy.  The
hits are compared bit for bit with those of the 8-wide tree, whose nodes, build
and traversal are its own."""
import ctypes
import itertools

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 9, 17, 130])
def test_small_trees(n):
    spec = scenes.hairball_scene(n, seed=n)
    rng = np.random.default_rng(n)
    # rays at the triangles' insides and past them, some with zero direction components
    tri = spec.tris[rng.integers(0, n, 600)]
    w = rng.dirichlet((2, 2, 2), 600)
    target = (tri * w[:, :, None]).sum(1) + np.where(rng.random((600, 1)) < 0.3, 0.3 * rng.normal(size=(600, 3)), 0.0)
    org = 3.0 * rng.normal(size=(600, 3))
    org[:60, :2] = target[:60, :2]
    org[60:90, 1:] = target[60:90, 1:]
    d = target - org
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    org, d = org.astype(np.float32), d.astype(np.float32)
    wide = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_W8,), leaf_size=1)
    want = wide.intersection(org, d, node_format=xtgpu.NODES_W8)
    wide.close()
    assert 0.5 < np.isfinite(want["t"]).mean() < 1.0
    keep = xtgpu.get_tuning()
    try:
        for leaf, layout, builder in itertools.product((1, 2, 3, 4), (0, 1), (0, 1)):
            xtgpu.set_tuning(node_layout=layout, bvh_builder=builder)
            sc = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_Q8), leaf_size=leaf)
            for fmt, variant in itertools.product((xtgpu.NODES_FP32, xtgpu.NODES_Q8), (0, 1, 2)):
                sc.set_tuning(extend_variant=variant)
                h = sc.intersection(org, d, node_format=fmt)
                np.testing.assert_array_equal(h.view(np.uint32), want.view(np.uint32))
            sc.close()
    finally:
        xtgpu.check(xtgpu.lib().xtgpu_set_tuning(ctypes.byref(keep)))
