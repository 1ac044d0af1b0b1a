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
#include <vector>
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
                                if (J.ufirst != 7) return 1;
                                // the ray of each path by enumeration: the v-th pair of pixel and
                                // position that a path of the wave has not had before
                                std::map<std::pair<int64_t, int64_t>, int64_t> seen;
                                std::vector<int64_t> ray_of;
                                for (int64_t p = first; p < first + count; ++p) {
                                    const int64_t s = p / npix, pix = p % npix;
                                    const std::pair<int64_t, int64_t> key(pix, lens ? s : s / spp1);
                                    if (!seen.count(key)) {
                                        const int64_t v = (int64_t)seen.size();
                                        if (v >= n || first + camera_ray_path(J, (int)v) != p) return 2;
                                        seen[key] = v;
                                    }
                                    ray_of.push_back(seen[key]);
                                    for (J.wide = 0; J.wide < 2; ++J.wide) {
                                        int smp;
                                        int64_t slot;
                                        sample_of(J, (int)(p - first), smp, slot);
                                        if (smp != s || slot != pix) return 3;
                                    }
                                    J.wide = 0;
                                }
                                if ((int64_t)seen.size() != n) return 4;
                                // the first shade pass takes every path once, those of one ray in a row
                                std::vector<char> taken((size_t)count, 0);
                                std::map<int64_t, int64_t> last;   // ray -> where its latest path was taken
                                for (int64_t i = 0; i < count; ++i) {
                                    int v = -1;
                                    const int64_t k = first_pass_path(J, (int)i, v);
                                    if (k < 0 || k >= count || taken[(size_t)k]) return 5;
                                    taken[(size_t)k] = 1;
                                    if (v != ray_of[(size_t)k]) return 6;
                                    if (last.count(v) && last[v] != i - 1) return 7;
                                    last[v] = i;
                                }
                                ++cases;
                            }
                    }
    // pixel slots: every pixel of the rectangle once, the tile's pixels in a row, and
    // the same pixels by 32-bit and by 64-bit division
    for (int tile = 0; tile <= 9; ++tile)
        for (int rw = 1; rw <= 20; rw += 3)
            for (int rh = 1; rh <= 20; rh += 3) {
                DevJob J{};
                J.x0 = 5; J.y0 = 11; J.rw = rw; J.rh = rh; J.tile = tile; J.spp1 = J.spp = 1; J.count = rw * rh;
                set_camera_rays(J, false, 0);
                std::vector<char> had((size_t)(rw * rh), 0);
                int px = 0, py = 0;
                for (int64_t k = 0; k < (int64_t)rw * rh; ++k) {
                    int x, y, wx, wy;
                    J.wide = 1;
                    pixel_of(J, k, wx, wy);
                    J.wide = 0;
                    pixel_of(J, k, x, y);
                    if (x != wx || y != wy || x < 5 || y < 11 || x >= 5 + rw || y >= 11 + rh) return 8;
                    char &h = had[(size_t)((y - 11) * rw + x - 5)];
                    if (h) return 9;
                    h = 1;
                    if (tile > 1 && k > 0 && ((x - 5) / tile != (px - 5) / tile || (y - 11) / tile != (py - 11) / tile))
                        if ((x - 5) % tile || (y - 11) % tile) return 10;   // a tile starts at its corner
                    px = x;
                    py = y;
                }
            }
    // division by multiplication at the ends of its range
    for (uint32_t d : {1u, 2u, 3u, 5u, 7u, 8u, 641u, 65535u, 65536u, 65537u, (1u << 30) - 1, 1u << 30, (1u << 31) - 1, 1u << 31})
        for (uint32_t n : {0u, 1u, d - 1, d, d + 1, 2 * d - 1, 3 * d, 12345678u, (1u << 26) + 1, (1u << 31) - 2, (1u << 31) - 1})
            if (n < (1u << 31) && fast_div(d).div(n) != n / d) return 11;
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
