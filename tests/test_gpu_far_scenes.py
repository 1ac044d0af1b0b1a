"""Box tests of all node formats where their arithmetic is strained: scenes far from the
origin along one axis, very large and very small ones (the triangle test's products of
three lengths stay below 2^127 up to 2^40), and a triangle so far away that plane
distances overflow on 8-wide nodes for rays with a zero or tiny direction component.
Hits that 64 bits show to be clearly inside a triangle and clearly the nearest must be
found."""
import dataclasses

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu
FORMATS = (xtgpu.NODES_FP32, xtgpu.NODES_Q8, xtgpu.NODES_W8)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("far,log2,outlier", [(0, 0, 0), (4096, 0, 0), (-4096, 0, 0), (4096, 36, 0), (4096, -30, 0),
                                              (0, 0, 60), (0, 36, 60), (-4096, 0, 100)])
def test_clear_hits_are_found(axis, far, log2, outlier):
    rng = np.random.default_rng(17 + axis)
    n, rays = 400, 3000
    scale = 2.0 ** log2
    tri = 10 * rng.random((n, 1, 3)) + rng.normal(size=(n, 3, 3))
    tri[:, :, axis] += far
    tri = (tri * scale).astype(np.float32)
    scene = tri
    if outlier:   # the root's quantum on this axis is 2^(outlier - 8)
        lone = np.zeros((1, 3, 3), np.float32)
        lone[0, 1, (axis + 1) % 3] = lone[0, 2, (axis + 2) % 3] = 1.0
        lone[0, :, axis] = 2.0 ** outlier
        scene = np.concatenate([tri, lone])
    spec = dataclasses.replace(scenes.hairball_scene(4, seed=1), tris=scene, obj_count=np.array([len(scene)], np.int32))
    k = rng.integers(0, n, rays)
    target = (tri[k].astype(np.float64) * rng.dirichlet((4, 4, 4), rays)[:, :, None]).sum(1)
    # origins a few units away; a third with one direction component zero, some with a tiny one
    step = rng.normal(size=(rays, 3)) * rng.uniform(1, 8, (rays, 1))
    step[: rays // 3, axis] = 0.0
    step[rays // 3: rays // 2, (axis + 1) % 3] = 0.0
    o = (target + step * scale).astype(np.float32)
    o[: rays // 3, axis] = target[: rays // 3, axis].astype(np.float32)
    d = target - o.astype(np.float64)
    d[: rays // 3, axis] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[: rays // 9, axis] = 1e-25
    d = d.astype(np.float32)
    # 64 bits: distances and the margin inside of every triangle
    O, D = o.astype(np.float64) / scale, d.astype(np.float64)
    T = tri.astype(np.float64) / scale
    e1, e2 = T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]
    nrm = np.cross(e1, e2)
    det = -D @ nrm.T
    s = O[:, None] - T[None, :, 0]
    q = np.cross(s, D[:, None])
    with np.errstate(divide="ignore", invalid="ignore"):
        t = (s * nrm).sum(2) / det
        u, v = (q * e2).sum(2) / det, -(q * e1).sum(2) / det
        margin = np.minimum(np.minimum(u, v), 1 - u - v)
    cos = np.abs(det) / np.linalg.norm(nrm, axis=1)
    t[~((margin > -0.05) & (t > -0.1))] = np.inf   # also what is nearly met
    first = np.argsort(t, axis=1)[:, :2]
    row = np.arange(rays)
    j = first[:, 0]
    extent = (T.max(1) - T.min(1)).min(1)
    # the point lies margin * extent inside the box on each axis: 0.01 at least, against coordinates'
    # roundings of 2^-12 at 4096
    clear = ((t[row, j] > 0.1) & np.isfinite(t[row, j]) & (margin[row, j] > 0.05) & (extent[j] > 0.2) &
             (cos[row, j] > 0.1) & (t[row, first[:, 1]] > t[row, j] + 0.1))
    assert clear.sum() > rays // 4
    sc = xtgpu.Scene(spec, node_formats=FORMATS, leaf_size=1)
    for fmt in FORMATS:
        h = sc.intersection(o, d, node_format=fmt)
        np.testing.assert_array_equal(h["prim"][clear], j[clear], err_msg=str(fmt))
    sc.close()
