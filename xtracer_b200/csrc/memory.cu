// Device and pinned memory that the entry points take and give back.
//
// cudaMalloc and cudaFree cost about 200 us each here (25 of each to load a scene,
// 10 of 16 ms), and the runtime's own pool hands everything back to the driver at
// every synchronisation, so the first cudaMallocAsync after one maps memory again
// (up to 0.5 ms in calls whose kernels take 20 us).  Freed blocks are kept here
// instead, up to KEEP_BYTES a device, the largest given back to the driver first; all
// of them when an allocation fails.
//
// A block is handed out only when nothing on the device uses it any more: dfree
// waits for the device, as cudaFree does, and dput is for blocks whose only users
// were on a stream that the caller has waited for.  So a block may go to another
// stream or thread next.
#include <cstring>
#include <list>
#include <map>
#include <mutex>
#include <unordered_map>

#include "xtgpu_internal.cuh"

namespace xtg {

namespace {

// One scene of 1M triangles with all three trees takes 0.7 GB; 0.5 % of the HBM.
constexpr size_t KEEP_BYTES = 1ull << 30;
// Pinned staging: blocks of up to STAGE_MAX bytes, STAGE_KEEP bytes kept.
constexpr size_t STAGE_KEEP = 32ull << 20;

struct Block {
    void *p;
    size_t cap;
    int dev;
};

struct Cache {
    std::mutex mu;
    std::unordered_map<void *, Block> live;
    std::list<Block> idle;
    std::map<int, size_t> kept;
    std::list<Block> pinned;
    size_t pinned_kept = 0;
};
// never destroyed: the driver may be gone before static destructors run
Cache &cache()
{
    static Cache *c = new Cache();
    return *c;
}

// sizes in steps of an eighth of their power of two, so that scenes of nearly one
// size use each other's blocks and at most an eighth is wasted
size_t size_class(size_t bytes)
{
    if (bytes <= 512) return 512;
    size_t step = 64;
    while (step * 16 < bytes) step <<= 1;
    return (bytes + step - 1) / step * step;
}

// Gives idle blocks of the device back to the driver until at most `keep` bytes are
// kept, the largest first: an allocation costs about as much whatever its size, and a
// program that loads one large scene after another finds all but its largest blocks.
void trim(Cache &c, int dev, size_t keep)
{
    while (c.kept[dev] > keep) {
        auto big = c.idle.end();
        for (auto it = c.idle.begin(); it != c.idle.end(); ++it)
            if (it->dev == dev && (big == c.idle.end() || it->cap > big->cap)) big = it;
        if (big == c.idle.end()) return;
        cudaFree(big->p);
        c.kept[dev] -= big->cap;
        c.idle.erase(big);
    }
}

}  // namespace

xtgpu_status dalloc(HostBuf &b, size_t bytes, cudaStream_t s)
{
    (void)s;
    dfree(b);
    int dev = 0;
    XTG_CUDA(cudaGetDevice(&dev));
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    Block k{nullptr, size_class(bytes), dev};
    auto best = c.idle.end();
    for (auto it = c.idle.begin(); it != c.idle.end(); ++it)
        if (it->dev == dev && it->cap >= k.cap && it->cap <= k.cap + k.cap / 4 &&
            (best == c.idle.end() || it->cap < best->cap))
            best = it;
    if (best != c.idle.end()) {
        k = *best;
        c.kept[dev] -= k.cap;
        c.idle.erase(best);
    } else {
        cudaError_t e = cudaMalloc(&k.p, k.cap);
        if (e == cudaErrorMemoryAllocation && c.kept[dev] > 0) {
            cudaGetLastError();
            trim(c, dev, 0);
            k.cap = bytes ? bytes : 16;
            e = cudaMalloc(&k.p, k.cap);
        }
        if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc", __FILE__, __LINE__);
    }
    c.live[k.p] = k;
    b.p = k.p;
    b.bytes = bytes;
    return XTGPU_OK;
}

void dput(HostBuf &b)
{
    if (!b.p) return;
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    auto it = c.live.find(b.p);
    if (it != c.live.end()) {
        const Block k = it->second;
        c.live.erase(it);
        c.idle.push_back(k);
        c.kept[k.dev] += k.cap;
        trim(c, k.dev, KEEP_BYTES);
    }
    b.p = nullptr;
    b.bytes = 0;
}

void dfree(std::initializer_list<HostBuf *> bufs)
{
    bool any = false;
    for (HostBuf *b : bufs) any = any || b->p;
    if (!any) return;
    // the blocks' device, which need not be the current one
    int dev = 0, now = 0;
    {
        Cache &c = cache();
        std::lock_guard<std::mutex> lock(c.mu);
        for (HostBuf *b : bufs)
            if (b->p && c.live.count(b->p)) dev = c.live[b->p].dev;
    }
    cudaGetDevice(&now);
    if (now != dev) cudaSetDevice(dev);
    cudaDeviceSynchronize();
    if (now != dev) cudaSetDevice(now);
    for (HostBuf *b : bufs) dput(*b);
}

void dfree(HostBuf &b) { dfree({&b}); }

xtgpu_status stage_get(HostBuf &b, size_t bytes)
{
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    Block k{nullptr, size_class(bytes < (64u << 10) ? (64u << 10) : bytes), 0};
    auto best = c.pinned.end();
    for (auto it = c.pinned.begin(); it != c.pinned.end(); ++it)
        if (it->cap >= k.cap && (best == c.pinned.end() || it->cap < best->cap)) best = it;
    if (best != c.pinned.end()) {
        k = *best;
        c.pinned_kept -= k.cap;
        c.pinned.erase(best);
    } else {
        XTG_CUDA(cudaHostAlloc(&k.p, k.cap, cudaHostAllocPortable));
    }
    c.live[k.p] = k;
    b.p = k.p;
    b.bytes = bytes;
    return XTGPU_OK;
}

void stage_put(HostBuf &b)
{
    if (!b.p) return;
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    const Block k = c.live[b.p];
    c.live.erase(b.p);
    c.pinned.push_back(k);
    c.pinned_kept += k.cap;
    while (c.pinned_kept > STAGE_KEEP) {
        cudaFreeHost(c.pinned.front().p);
        c.pinned_kept -= c.pinned.front().cap;
        c.pinned.pop_front();
    }
    b.p = nullptr;
    b.bytes = 0;
}

// One byte in every page of a result that is about to be written, so that a fresh
// buffer's page faults (about 0.25 us each, 300 for a 320x240 frame) run while the
// GPU works.
void touch_pages(void *p, size_t bytes)
{
    volatile char *q = (volatile char *)p;
    for (size_t i = 0; i < bytes; i += 4096) q[i] = q[i];
    if (bytes) q[bytes - 1] = q[bytes - 1];
}

}  // namespace xtg
