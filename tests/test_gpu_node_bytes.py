"""Memory of the FP32 and Q8 trees: a place for each four-child node that a walk can
reach and none for the others, in either node order, by either builder."""
import ctypes

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu


def reached(left, right, leaf):
    """Inner nodes of the exported hierarchy an even number of levels below the root with more than `leaf` primitives."""
    n = len(left)
    if n == 0:
        return 0
    order, depth = [0], {0: 0}
    for i in order:
        for c in (left[i], right[i]):
            if c >= 0:
                depth[c] = depth[i] + 1
                order.append(c)
    prims = {}
    for i in reversed(order):
        prims[i] = sum(1 if c < 0 else prims[c] for c in (left[i], right[i]))
    return sum(depth[i] % 2 == 0 and prims[i] > leaf for i in order)


@pytest.mark.parametrize("n", [1, 2, 3, 5, 1025, 4000])
def test_node_bytes(n):
    spec = scenes.hairball_scene(n, seed=n)
    keep = xtgpu.get_tuning()
    try:
        for leaf, layout, builder in ((1, 1, 0), (1, 0, 0), (2, 1, 1), (3, 0, 1), (4, 1, 0)):
            xtgpu.set_tuning(node_layout=layout, bvh_builder=builder)
            sc = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_Q8), leaf_size=leaf)
            b = sc.bvh_export()
            nodes = max(1, reached(b["left"].tolist(), b["right"].tolist(), leaf))   # a tree of one leaf has a dummy
            assert b["info"].node_bytes_fp32 == 128 * nodes
            assert b["info"].node_bytes_q8 == 64 * nodes
            assert sc.device_bytes() > 192 * nodes
            sc.close()
    finally:
        xtgpu.check(xtgpu.lib().xtgpu_set_tuning(ctypes.byref(keep)))
