"""Host entry points on ordinary, pinned and managed memory: small results are staged through the library's own
pinned blocks, whatever the caller's buffer is."""
import ctypes as C

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu


def managed(n):
    rt = C.CDLL("libcudart.so.12")
    p = C.c_void_p()
    assert rt.cudaMallocManaged(C.byref(p), C.c_size_t(4 * n), 1) == 0
    return p, np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (n,)), lambda: rt.cudaFree(p)


@pytest.mark.parametrize("n", [333, 100_000])   # staged, and copied by the driver
def test_trace_and_render(n):
    import torch
    sc = xtgpu.Scene(scenes.hairball_scene(5000, seed=4))
    rng = np.random.default_rng(n)
    o = np.zeros((n, 4), np.float32)
    o[:, :3] = 3 * rng.normal(size=(n, 3))
    d = np.zeros((n, 4), np.float32)
    d[:, :3] = -o[:, :3] / np.linalg.norm(o[:, :3], axis=1, keepdims=True)
    d[:, 3] = np.inf
    p = xtgpu.RenderParams(xtgpu.AO, n // 3, 3, 1, 2, 1.0, 8, 0, 0, 0, 0, 0, 1, 0)
    results = []
    for kind in ("ordinary", "pinned", "managed"):
        if kind == "managed":
            frees, bufs = [], []
            for _ in range(3):
                _, a, free = managed(4 * n)
                bufs.append(a)
                frees.append(free)
        else:
            bufs = [torch.zeros(4 * n, dtype=torch.float32, pin_memory=kind == "pinned").numpy() for _ in range(3)]
            frees = []
        bufs[0][:], bufs[1][:], bufs[2][:] = o.ravel(), d.ravel(), 0
        ptr = [C.c_void_p(b.ctypes.data) for b in bufs]
        xtgpu.check(xtgpu.lib().xtgpu_trace_host(sc.handle, n, ptr[0], ptr[1], ptr[2], 0, None))
        hits = bufs[2].copy()
        rays = C.c_uint64()
        xtgpu.check(xtgpu.lib().xtgpu_render_host(sc.handle, C.byref(p), ptr[2], C.byref(rays), None))
        frame = bufs[2][:4 * 3 * (n // 3)].copy()
        results.append((hits.view(np.uint32), frame.view(np.uint32), rays.value))
        torch.cuda.synchronize()
        del bufs
        for free in frees:
            free()
    for r in results[1:]:
        np.testing.assert_array_equal(r[0], results[0][0])
        np.testing.assert_array_equal(r[1], results[0][1])
        assert r[2] == results[0][2]
    sc.close()
