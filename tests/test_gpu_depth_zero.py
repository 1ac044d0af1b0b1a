"""A pathtracer job of depth 0 beside jobs that have passes: the frame and the ray
count are those of the job alone (black, no ray followed), wherever its paths fall
in the waves."""
import numpy as np
import pytest

from xtracer_b200 import scenes, xtgpu
from xtracer_b200.service import Service

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("merge", [False, True])
@pytest.mark.parametrize("wave", [1 << 20, 777])
def test_depth_zero_in_a_mix(wave, merge):
    sc = xtgpu.Scene(scenes.uv_scene())   # a sky and spheres that glow
    w, h, spp = 40, 30, 3
    # both are in view
    assert sc.render(xtgpu.EMISSION, w, h)[0][..., :3].any() and (sc.render(xtgpu.STENCIL, w, h)[0][..., 3] == 0).any()
    svc = Service([sc], wave_paths=wave, merge_jobs=merge)
    depths = (0, 4, 0, 1)
    ids = [svc.submit(0, xtgpu.PATHTRACER, w, h, spp, d, seed=5 + k) for k, d in enumerate(depths)]
    svc.run()
    total = 0
    for k, (jid, d) in enumerate(zip(ids, depths)):
        alone, rays = sc.render(xtgpu.PATHTRACER, w, h, spp, d, seed=5 + k)
        if d == 0:
            assert rays == 0 and not alone[..., :3].any()
        np.testing.assert_array_equal(svc.result(jid).view(np.uint32), alone.view(np.uint32))
        assert svc.poll(jid).rays == rays
        total += rays
    assert svc.stats().rays == total
    svc.close()
    sc.close()
