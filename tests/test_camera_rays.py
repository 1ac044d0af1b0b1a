"""Camera rays shared between the samples of one position (xtracer_b200/csrc/
wavefront.cuh): the numbering of a wave's rays against a plain enumeration, on
the CPU, and the frames of waves cut anywhere against whole frames, on the GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from xtracer_b200 import build, scenes

CHECK = r"""
#include <cstdio>
#include <map>
#include <utility>
#include "wavefront.cuh"
using namespace xtg;
int main()
{
    long cases = 0;
    for (int rw = 1; rw <= 5; rw += 2)
        for (int rh = 1; rh <= 3; ++rh)
            for (int spp1 = 1; spp1 <= 4; ++spp1)
                for (int P = 1; P <= 4; P += P < 2 ? 1 : 2)
                    for (int lens = 0; lens < 2; ++lens) {
                        DevJob J{};
                        J.rw = rw; J.rh = rh; J.spp1 = spp1; J.spp = P * spp1;
                        const int64_t npix = rw * rh, paths = npix * J.spp;
                        for (int64_t first = 0; first < paths; ++first)
                            for (int64_t count = 1; first + count <= paths; ++count) {
                                J.first = first; J.count = count;
                                const int64_t n = set_camera_rays(J, lens, 7);
                                std::map<std::pair<int64_t, int64_t>, int64_t> seen;   // (pixel, position) -> ray
                                for (int64_t p = first; p < first + count; ++p) {
                                    const int64_t s = p / npix, pix = p % npix;
                                    const int64_t v = camera_ray_of(J, npix, p, s, pix);
                                    const std::pair<int64_t, int64_t> key(pix, lens ? s : s / spp1);
                                    if (v < 0 || v >= n || J.ufirst != 7) return 1;
                                    if (!seen.count(key)) {
                                        if ((int64_t)seen.size() != v) return 2;   // numbered in path order
                                        if (camera_ray_path(J, npix, v) != p) return 3;
                                        seen[key] = v;
                                    } else if (seen[key] != v) return 4;
                                }
                                if ((int64_t)seen.size() != n) return 5;
                                // the first shade pass takes every path once, those of one ray in a row
                                std::map<int64_t, bool> taken;
                                std::map<int64_t, int64_t> last;   // ray -> where its latest path was taken
                                for (int64_t i = 0; i < count; ++i) {
                                    const int64_t k = first_pass_path(J, npix, i), p = first + k;
                                    if (k < 0 || k >= count || taken.count(k)) return 6;
                                    taken[k] = true;
                                    const int64_t v = camera_ray_of(J, npix, p, p / npix, p % npix);
                                    if (last.count(v) && last[v] != i - 1) return 7;
                                    last[v] = i;
                                }
                                ++cases;
                            }
                    }
    printf("%ld\n", cases);
    return 0;
}
"""


@pytest.mark.skipif(not (shutil.which(build.NVCC) or os.path.exists(build.NVCC)), reason="no nvcc")
def test_ray_numbering(tmp_path):
    src = tmp_path / "check.cu"
    src.write_text(CHECK)
    exe = str(tmp_path / "check")
    subprocess.run([build.NVCC] + build.CCBIN + ["-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I" + build.CSRC, "-o", exe,
                    str(src)], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and int(r.stdout) > 10000, (r.returncode, r.stdout)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("aa,dist,spp", [(1, 0, 7), (2, 0, 3), (3, 1, 4)])
def test_waves_cut_anywhere(aa, dist, spp, lens):
    """Waves that end inside a sample, a position or a run of samples give the frame and the ray count of one
    wave, and samples taken together those of samples taken one a wave."""
    from xtracer_b200 import xtgpu
    spec = scenes.spheres_scene(24, seed=3)
    if lens:
        spec.camera.flength, spec.camera.aperture = 12.0, 0.5
    sc = xtgpu.Scene(spec, node_formats=(xtgpu.NODES_FP32, xtgpu.NODES_W8), leaf_size=1)
    w, h = 45, 31
    for integ in (xtgpu.PATHTRACER, xtgpu.AO, xtgpu.DEPTH):
        for fmt in (xtgpu.NODES_FP32, xtgpu.NODES_W8):
            sc.set_tuning(wave_paths=1 << 22)
            whole, rays = sc.render(integ, w, h, spp, 3, 5.0, 9, fmt, aa=aa, distribution=dist)
            for wave in (1024, w * h, 2 * w * h + 1, spp * w * h - 17):
                sc.set_tuning(wave_paths=wave)
                cut, r = sc.render(integ, w, h, spp, 3, 5.0, 9, fmt, aa=aa, distribution=dist)
                assert r == rays
                np.testing.assert_array_equal(cut, whole)
    sc.close()
