"""Scenes opened and closed while another thread captures a graph, and what a closed
scene's blocks wait for (xtracer_b200/csrc/memory.cu, wait_device)."""
import threading

import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu

pytestmark = pytest.mark.gpu


def on_a_thread(work):
    bad = []

    def body():
        try:
            work()
        except Exception as e:
            bad.append(e)

    t = threading.Thread(target=body)
    t.start()
    t.join()
    assert not bad, bad


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_scenes_beside_a_capture(mode):
    """What the calls of another thread do leaves the capture whole, and their results are the usual ones."""
    import torch
    spec = scenes.hairball_scene(3000, seed=2)
    sc = xtgpu.Scene(spec)
    want = sc.render(xtgpu.AO, 40, 30, 2, seed=5)[0]
    x = torch.arange(1024, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    got = []

    def work():
        torch.cuda.set_device(0)
        stream = torch.cuda.Stream()
        for formats in ((xtgpu.NODES_FP32,), (xtgpu.NODES_FP32, xtgpu.NODES_W8)):
            other = xtgpu.Scene(spec, node_formats=formats, leaf_size=1, stream=stream)
            other.close()
        got.append(sc.render(xtgpu.AO, 40, 30, 2, seed=5)[0])
        sc.close()

    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s, capture_error_mode=mode):
        y = x * 2
        on_a_thread(work)
        z = y + 1
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(z.cpu().numpy(), 2 * np.arange(1024, dtype=np.float32) + 1)
    np.testing.assert_array_equal(got[0], want)


def test_close_waits_for_the_device():
    """A closed scene's blocks are free only when all streams have run: after close() nothing that was enqueued
    before it is still running."""
    import torch
    sc = xtgpu.Scene(scenes.hairball_scene(3000, seed=2))
    s, e = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)   # some 10 ms
        e.record(s)
    assert not e.query()
    sc.close()
    assert e.query()
