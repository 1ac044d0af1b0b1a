"""Blocks kept between calls (xtracer_b200/csrc/memory.cu): results where the
staged copies give way to the driver's, scenes loaded and closed by several
threads at once, and how much stays allocated."""
import threading

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu
STAGE_MAX = 4 << 20   # bytes


def rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(n, 3)) * 3.0
    d = -o + 0.5 * rng.normal(size=(n, 3))
    return o.astype(np.float32), (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 31, STAGE_MAX // 48, STAGE_MAX // 48 + 1, 200_001])
def test_host_batches(n):
    import torch
    sc = xtgpu.Scene(scenes.hairball_scene(5000, seed=4))
    o, d = rays(n, n)
    got = sc.intersection(o, d, tmin=0.25, tmax=5.0)
    org, dirs = torch.empty((n, 4), device="cuda"), torch.empty((n, 4), device="cuda")
    org[:, :3], org[:, 3] = torch.from_numpy(o).cuda(), 0.25
    dirs[:, :3], dirs[:, 3] = torch.from_numpy(d).cuda(), 5.0
    hits = torch.empty((n, 4), device="cuda")
    xtgpu.check(xtgpu.lib().xtgpu_trace(sc.handle, n, org.data_ptr(), dirs.data_ptr(), hits.data_ptr(), 0, None))
    np.testing.assert_array_equal(got.view(np.uint32).reshape(n, 4), hits.cpu().numpy().view(np.uint32))
    sc.close()


@pytest.mark.parametrize("w,h", [(512, 512), (513, 512), (1, 1)])
def test_host_frames(w, h):
    import ctypes

    import torch
    sc = xtgpu.Scene(scenes.spheres_scene(16, seed=4))
    img, n = sc.render(xtgpu.PATHTRACER, w, h, 2, 3, seed=8)
    p = xtgpu.RenderParams(xtgpu.PATHTRACER, w, h, 2, 3, 100.0, 8, 0, 0, 0, 0, 0, 1, 0)
    out, r = torch.full((h, w, 4), -7.0, device="cuda"), ctypes.c_uint64()
    xtgpu.check(xtgpu.lib().xtgpu_render(sc.handle, ctypes.byref(p), out.data_ptr(), ctypes.byref(r), None))
    assert r.value == n
    np.testing.assert_array_equal(img, out.cpu().numpy())
    sc.close()


def test_scenes_from_several_threads():
    sizes = (300, 5000, 5100, 40_000)
    specs = [scenes.hairball_scene(n, seed=n) for n in sizes]
    o, d = rays(3000, 1)
    want = []
    for sp in specs:
        sc = xtgpu.Scene(sp, node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_W8), leaf_size=1)
        want.append((sc.intersection(o, d, node_format=xtgpu.NODES_W8), sc.render(xtgpu.AO, 64, 48, 4, seed=3)[0]))
        sc.close()
    bad = []

    def work(k):
        import torch
        stream = torch.cuda.Stream()
        for _ in range(6):
            sc = xtgpu.Scene(specs[k], node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_W8), leaf_size=1,
                             stream=stream if k % 2 else None)
            h = sc.intersection(o, d, node_format=xtgpu.NODES_W8)
            img = sc.render(xtgpu.AO, 64, 48, 4, seed=3)[0]
            sc.close()
            if not (np.array_equal(h.view(np.uint32), want[k][0].view(np.uint32)) and np.array_equal(img, want[k][1])):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(specs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_what_stays_allocated_is_bounded():
    import torch
    sc = xtgpu.Scene(scenes.hairball_scene(10, seed=1))
    sc.render(xtgpu.DEPTH, 64, 64)
    sc.close()
    before = torch.cuda.mem_get_info()[0]
    spec = scenes.terrain_scene(3_000_000, seed=1)
    sc = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_W8), leaf_size=1)
    assert sc.device_bytes() > 1 << 30   # more than is kept
    sc.close()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= (1 << 30) + (64 << 20)
