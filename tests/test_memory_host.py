"""The block cache (xtracer_b200/csrc/memory.cu) on the CPU, linked with a stand-in
for the CUDA runtime whose waits and allocations can be made to fail."""
import os
import shutil
import subprocess

import pytest

from xtracer_b200 import build

FAKE = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <string>
#include "xtgpu_internal.cuh"

static size_t capacity = ~(size_t)0, used = 0;
static std::map<void *, size_t> device, host;
static bool refuse_waits = false;   // as while another thread captures a stream
static int waits = 0, device_syncs = 0, current = 0;
static cudaError_t last = cudaSuccess;
static cudaError_t fail(cudaError_t e) { return last = e; }

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    if (used + n > capacity) return fail(cudaErrorMemoryAllocation);
    *p = std::malloc(16);
    device[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p)
{
    if (!p) return cudaSuccess;
    if (!device.count(p)) return fail(cudaErrorInvalidValue);
    ++waits;
    if (refuse_waits) return fail(cudaErrorStreamCaptureUnsupported);
    used -= device[p];
    device.erase(p);
    return cudaSuccess;   // the address is not given to malloc again: tests compare addresses
}
static bool refuse_pinning = false;
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    if (refuse_pinning) return fail(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    host[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { host.erase(p); return cudaSuccess; }
static cudaError_t wait() { ++waits; return refuse_waits ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { ++device_syncs; return wait(); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return wait(); }
cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    if (p == (void *)16) return fail(cudaErrorInvalidValue);
    a->type = device.count((void *)p) ? cudaMemoryTypeDevice : host.count((void *)p) ? cudaMemoryTypeHost
              : p == (void *)32 ? cudaMemoryTypeManaged : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t) { return ""; }
}

namespace xtg {
void set_error(const std::string &) {}
xtgpu_status cuda_fail(cudaError_t e, const char *, const char *, int)
{
    return e == cudaErrorMemoryAllocation ? XTGPU_ERR_NOMEM : XTGPU_ERR_CUDA;
}
}  // namespace xtg
using namespace xtg;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
"""

REFUSED_WAITS = r"""
int main()
{
    HostBuf a, b, c;
    // an ordinary block comes back
    CHECK(dalloc(a, 1000, 0) == XTGPU_OK);
    void *p = a.p;
    dfree(a);
    CHECK(!a.p && waits == 1 && device.size() == 3);   // the block and the two of a wait
    CHECK(dalloc(a, 1000, 0) == XTGPU_OK && a.p == p);
    // one whose wait was refused does not, and leaves no error behind
    refuse_waits = true;
    dfree(a);
    CHECK(!a.p && last == cudaSuccess);
    CHECK(dalloc(b, 1000, 0) == XTGPU_OK && b.p != p);
    void *p2 = b.p;
    // the same for the blocks of a call and of a build, and for staging
    { Scratch s; s.b = b; b = HostBuf(); }
    CHECK(dalloc(b, 1000, 0) == XTGPU_OK && b.p != p && b.p != p2);
    void *p3 = b.p;
    dput(b);   // waited for by its caller
    void *p4;
    {
        Tmp t{0};
        float *f;
        CHECK(t.get(&f, 250) == XTGPU_OK);
        p4 = f;
        CHECK(p4 == p3);
    }
    CHECK(last == cudaSuccess);
    CHECK(dalloc(b, 1000, 0) == XTGPU_OK && b.p != p && b.p != p2 && b.p != p4);
    void *h;
    { Stage s; CHECK(stage_get(s.b, 100) == XTGPU_OK); h = s.b.p; }
    CHECK(last == cudaSuccess);
    HostBuf st;
    CHECK(stage_get(st, 100) == XTGPU_OK && st.p != h);
    // a wait that succeeds makes all of them idle
    refuse_waits = false;
    dfree(b);
    std::set<void *> got;
    for (int i = 0; i < 4; ++i) {
        HostBuf x;
        CHECK(dalloc(x, 1000, 0) == XTGPU_OK);
        got.insert(x.p);
    }
    CHECK(got.count(p) && got.count(p2) && got.count(p4));
    HostBuf st2;
    CHECK(stage_get(st2, 100) == XTGPU_OK && st2.p == h);
    // the wait of one device says nothing about another's blocks
    current = 1;
    CHECK(dalloc(c, 1000, 0) == XTGPU_OK);
    void *q = c.p;
    refuse_waits = true;
    dfree(c);
    refuse_waits = false;
    current = 0;
    CHECK(dalloc(a, 5000, 0) == XTGPU_OK);
    dfree(a);
    current = 1;
    CHECK(dalloc(c, 1000, 0) == XTGPU_OK && c.p != q);
    dfree(c);
    CHECK(current == 1);
    // none of these waits was one that other threads' captures do not survive
    CHECK(device_syncs == 0);
    return 0;
}
"""

NO_MEMORY = r"""
int main()
{
    // with nothing left to allocate, a block is still waited for and given back
    HostBuf a;
    CHECK(dalloc(a, 1 << 20, 0) == XTGPU_OK);
    void *p = a.p;
    capacity = used;
    dfree(a);
    CHECK(last == cudaSuccess && waits == 1);
    CHECK(dalloc(a, 1 << 20, 0) == XTGPU_OK && a.p == p);
    return 0;
}
"""


def run(tmp_path, body):
    (tmp_path / "check.cpp").write_text(FAKE + body)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    exe = str(tmp_path / "check")
    subprocess.run([gxx, "-std=c++17", "-O1", "-x", "c++", "-I" + build.CSRC, "-I" + cuda, "-o", exe,
                    str(tmp_path / "check.cpp"), os.path.join(build.CSRC, "memory.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


pytestmark = pytest.mark.skipif(not os.path.exists(build.NVCC) or not (shutil.which("g++") or os.path.exists("/usr/bin/g++")),
                                reason="no CUDA headers or host compiler")


EXACT_SIZE = r"""
int main()
{
    // a request that fits, although its size class does not, with nothing idle to give back
    HostBuf a, b;
    capacity = 1000 * 1024 + 1;
    CHECK(dalloc(a, capacity, 0) == XTGPU_OK && a.bytes == capacity && used == capacity && last == cudaSuccess);
    CHECK(dalloc(b, 1, 0) == XTGPU_ERR_NOMEM && !b.p);
    return 0;
}
"""

POOL = r"""
int main()
{
    // idle blocks make room for the library's stream-ordered allocations
    HostBuf a;
    CHECK(dalloc(a, 64 << 20, 0) == XTGPU_OK);
    dfree(a);
    capacity = used + 1024;
    void *p = nullptr;
    CHECK(pool_get(&p, 32 << 20, 0) == XTGPU_OK && p && last == cudaSuccess);
    void *q = &capacity;
    CHECK(pool_get(&q, 64 << 20, 0) == XTGPU_ERR_NOMEM && !q);
    return 0;
}
"""

RELEASE = r"""
int main()
{
    HostBuf a, b, c, st;
    const size_t before = used;
    CHECK(dalloc(a, 1 << 20, 0) == XTGPU_OK && dalloc(b, 2 << 20, 0) == XTGPU_OK && stage_get(st, 100) == XTGPU_OK);
    stage_put(st, true);
    dfree(a);
    current = 1;
    CHECK(dalloc(c, 4 << 20, 0) == XTGPU_OK);
    refuse_waits = true;
    dfree(c);                       // held
    refuse_waits = false;
    current = 0;
    const size_t in_use = device[b.p];
    uint64_t bytes = 0;
    CHECK(xtgpu_release_memory(&bytes) == XTGPU_OK && bytes >= 5u << 20 && host.empty() && current == 0);
    CHECK(device.count(b.p) && used <= before + in_use + 4 * 512);   // b, and the blocks of two waits
    CHECK(xtgpu_release_memory(nullptr) == XTGPU_OK);
    // refused: what is idle stays idle
    dfree(b);
    refuse_waits = true;
    CHECK(xtgpu_release_memory(&bytes) == XTGPU_OK && bytes == 0 && last == cudaSuccess);
    refuse_waits = false;
    CHECK(xtgpu_release_memory(&bytes) == XTGPU_OK && bytes == in_use);
    return 0;
}
"""

KINDS = r"""
int main()
{
    // what host code may stage: everything but device memory and what the driver cannot name
    HostBuf d, h;
    int x = 0;
    CHECK(dalloc(d, 64, 0) == XTGPU_OK && stage_get(h, 64) == XTGPU_OK);
    CHECK(!host_memory(d.p) && host_memory(h.p) && host_memory(&x) && host_memory((void *)32));
    CHECK(!host_memory((void *)16) && last == cudaSuccess);
    return 0;
}
"""

UNPINNED = r"""
int main()
{
    // staging that cannot be pinned is ordinary memory, and is not kept
    refuse_pinning = true;
    HostBuf a;
    CHECK(stage_get(a, 100000) == XTGPU_OK && a.bytes == 100000 && last == cudaSuccess);
    ((char *)a.p)[99999] = 1;
    stage_put(a, true);
    refuse_waits = true;
    { Stage s; CHECK(stage_get(s.b, 100) == XTGPU_OK); }
    refuse_waits = false;
    refuse_pinning = false;
    CHECK(stage_get(a, 100) == XTGPU_OK && host.count(a.p));
    return 0;
}
"""


@pytest.mark.parametrize("body", [REFUSED_WAITS, NO_MEMORY, EXACT_SIZE, POOL, RELEASE, KINDS, UNPINNED],
                         ids=["refused", "no_memory", "exact_size", "pool", "release", "kinds", "unpinned"])
def test_cache(tmp_path, body):
    run(tmp_path, body)
