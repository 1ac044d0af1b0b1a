"""The 8-wide collapse after an error (xtracer_b200/csrc/wide.cuh, wide_level_nodes), on
the CPU: a dozen levels are launched between two looks of the host, so a level that
follows a node without room must read nothing."""
import os
import re
import subprocess

import pytest

from xtracer_b200 import build

CHECK = r"""
#include <cstdio>
#include "wide.cuh"
using namespace xtg;
int main()
{
    const int max_nodes = 100, levels = 6;
    for (int fail_at = -1; fail_at < levels; ++fail_at) {
        int ctr[4 + levels + 1] = {1, 0, 0, 0, 1};
        int written[levels + 1] = {1};   // items of each level that are there to be read
        for (int l = 0; l < levels; ++l) {
            const int n = wide_level_nodes(ctr, l, max_nodes);
            if (n < 0 || n > written[l]) { std::printf("level %d reads %d of %d\n", l, n, written[l]); return 1; }
            if (fail_at < 0 && n != written[l]) { std::printf("level %d stops\n", l); return 1; }
            for (int i = 0; i < n; ++i) {
                const int ni = l < 2 ? 4 : 1;
                ctr[4 + l + 1] += ni;             // as k_wide_level: counted first,
                if (l == fail_at && i == n - 1) {
                    ctr[4 + l + 1] += max_nodes;  // (a count past what the arrays hold)
                    ctr[2] = 1;                   // then found to have no room
                } else {
                    written[l + 1] += ni;
                }
            }
        }
    }
    // a count that is not one of nodes, without the flag
    int ctr[5] = {1, 0, 0, 0, max_nodes + 1};
    if (wide_level_nodes(ctr, 0, max_nodes) != 0) return 2;
    ctr[4] = -1;
    if (wide_level_nodes(ctr, 0, max_nodes) != 0) return 3;
    ctr[4] = max_nodes;
    return wide_level_nodes(ctr, 0, max_nodes) == max_nodes ? 0 : 4;
}
"""


@pytest.mark.skipif(not os.path.exists(build.NVCC), reason="no nvcc")
def test_levels_after_an_error_read_nothing(tmp_path):
    # the kernel takes its count there, and nowhere else
    src = open(os.path.join(build.CSRC, "wide.cu")).read()
    body = src[src.index("    k_wide_level("):src.index("xtgpu_status build_wide")]
    assert "wide_level_nodes(ctr, level, max_nodes)" in body and not re.search(r"=\s*ctr\[4 \+ level\]", body)
    (tmp_path / "check.cu").write_text(CHECK)
    exe = str(tmp_path / "check")
    subprocess.run([build.NVCC] + build.CCBIN + ["-std=c++17", "--expt-relaxed-constexpr", "-I" + build.CSRC, "-o", exe,
                    str(tmp_path / "check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
