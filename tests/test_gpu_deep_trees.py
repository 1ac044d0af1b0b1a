"""Traversal stacks at their bounds: hierarchies as deep as Morton codes make them (a
chain of 30 splits, and one with equal codes below it), all of whose boxes every ray
meets, so that each visit pushes what it can.  48 entries hold FP32 and Q8 trees of
depth 30, 96 deeper ones; 32 and 64 the 8-wide trees."""
import dataclasses

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu
FORMATS = (xtgpu.NODES_FP32, xtgpu.NODES_Q8, xtgpu.NODES_W8)
R = 2048.0   # half a triangle's box; the centroids lie in [0, 1024)


def chain(copies, seed):
    """One triangle for each bit of the code (a power of two on one axis), the far corner, and `copies` more in the
    first cell: splits one after another, then equal codes.  Every triangle's box is centred on its cell and reaches
    past all the others' centres."""
    rng = np.random.default_rng(seed)
    c = [np.full(3, 1023.0), np.zeros(3)]
    for j in range(10):
        for a in range(3):
            p = np.zeros(3)
            p[a] = 2.0 ** j
            c.append(p)
    c = np.array(c + [np.zeros(3)] * copies) + rng.integers(0, 16, (32 + copies, 3)) / 64.0
    c[0], c[1] = 1023.0, 0.0   # the centroids' bounds: cells of (nearly) unit size
    # the box's corners at the ends of one edge; the third corner anywhere inside
    s = rng.choice([-1.0, 1.0], (len(c), 3))
    t = np.stack([c + R * s, c - R * s, c + rng.integers(-1500, 1500, (len(c), 3))], axis=1)
    return t[rng.permutation(len(t))].astype(np.float32)


@pytest.mark.parametrize("copies", [0, 70, 300])
def test_deep_trees(copies):
    tris = chain(copies, 5 + copies)
    spec = dataclasses.replace(scenes.hairball_scene(4, seed=1), tris=tris, obj_count=np.array([len(tris)], np.int32))
    rng = np.random.default_rng(9)
    n = 4000
    o = (500 * rng.normal(size=(n, 3))).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d[:200] = np.eye(3)[rng.integers(0, 3, 200)] * rng.choice([-1.0, 1.0], (200, 1))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    sc = xtgpu.Scene(spec, node_formats=FORMATS, leaf_size=1)
    depth = sc.bvh_export()["info"].depth
    assert depth > 30 if copies else 25 <= depth <= 30
    hits = {}
    for fmt in FORMATS:
        for variant in (0, 2):
            for entries in (0, 32, 64):
                sc.set_tuning(extend_variant=variant, stack_entries=entries)
                hits[fmt, variant, entries] = sc.intersection(o, d, node_format=fmt).copy()
    sc.close()
    first = hits[xtgpu.NODES_W8, 2, 0]
    for k, h in hits.items():
        np.testing.assert_array_equal(h.view(np.uint32), first.view(np.uint32), err_msg=str(k))
    # against 64 bits: what is clearly the nearest, met clearly inside and not edge-on
    v0, e1, e2 = (tris[:, 0].astype(np.float64), (tris[:, 1] - tris[:, 0]).astype(np.float64),
                  (tris[:, 2] - tris[:, 0]).astype(np.float64))
    checked = 0
    for i in range(n):
        oo, dd = o[i].astype(np.float64), d[i].astype(np.float64)
        nrm = np.cross(e1, e2)
        det = -nrm @ dd
        s = oo - v0
        q = np.cross(s, dd)
        with np.errstate(divide="ignore", invalid="ignore"):
            t = (nrm * s).sum(1) / det
            u, v = (e2 * q).sum(1) / det, -(e1 * q).sum(1) / det
            margin = np.minimum(np.minimum(u, v), 1 - u - v)
            cos = np.abs(det) / np.linalg.norm(nrm, axis=1)
        near = (margin > -1e-3) & (t > -1.0)
        if not near.any():
            assert first["prim"][i] == 0xFFFFFFFF
            continue
        k = np.flatnonzero(near)
        k = k[np.argsort(t[k])]
        j = k[0]
        clear = margin[j] > 1e-3 and t[j] > 1.0 and cos[j] > 0.05 and (len(k) == 1 or t[k[1]] > t[j] + 1.0)
        if clear:
            checked += 1
            assert first["prim"][i] == j
            # coordinates below 2^12 relative to the origin, some sixteen roundings, over the cosine
            assert abs(first["t"][i] - t[j]) <= 16 * 2.0 ** -24 * 4096 / cos[j]
    assert checked > n // 4
