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
// stream or thread next.  A wait can be refused (while another thread captures a stream
// in the global mode): the blocks are then held until a later wait succeeds, and are
// nobody's meanwhile.
#include <cstdlib>
#include <cstring>
#include <iterator>
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
    bool pageable = false;   // a staging block that could not be pinned
};

struct Cache {
    std::mutex mu;
    std::unordered_map<void *, Block> live;
    std::list<Block> idle;
    std::map<int, size_t> kept;
    std::list<Block> pinned;
    size_t pinned_kept = 0;
    // given back, but what used them has not been waited for: device and pinned blocks,
    // the latter with the device that was current
    std::list<Block> held, held_pinned;
    // wait_device: blocks to free, as many as threads have waited at once, and one that stays
    std::map<int, std::list<void *>> tokens;
    std::map<int, void *> anchor;
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
        if (cudaFree(big->p) != cudaSuccess) {   // refused (a capture in the global mode): it stays idle
            cudaGetLastError();
            return;
        }
        c.kept[dev] -= big->cap;
        c.idle.erase(big);
    }
}

void keep_idle(Cache &c, const Block &k)
{
    c.idle.push_back(k);
    c.kept[k.dev] += k.cap;
    trim(c, k.dev, KEEP_BYTES);
}

void keep_pinned(Cache &c, const Block &k)
{
    if (k.pageable) {
        free(k.p);
        return;
    }
    c.pinned.push_back(k);
    c.pinned_kept += k.cap;
    while (c.pinned_kept > STAGE_KEEP) {
        cudaFreeHost(c.pinned.front().p);
        c.pinned_kept -= c.pinned.front().cap;
        c.pinned.pop_front();
    }
}

// The blocks of one device taken out of a list.
std::list<Block> take_of(std::list<Block> &from, int dev)
{
    std::list<Block> out;
    for (auto it = from.begin(); it != from.end();) {
        auto next = std::next(it);
        if (it->dev == dev) out.splice(out.end(), from, it);
        it = next;
    }
    return out;
}

void *small_block()
{
    void *p = nullptr;
    if (cudaMalloc(&p, 512) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}

// Waits for everything on the device, as cudaFree does, by cudaFree of a small block.
// cudaDeviceSynchronize would do, but is refused while any stream of the device is being
// captured, in whatever mode, and the capture is lost by it: closing a scene would
// break the graph that a service, or the caller, captures on another thread.  Another
// small block, never freed, keeps the memory behind it mapped, and the block to free next
// is allocated at once, in the place of the last: 3.1 us to free on an idle device and 1.5
// to allocate (cudaDeviceSynchronize 3.3; 260 and 330 where the memory is mapped anew).
// Once a wait has succeeded, what was held before it began is idle.  A refused wait's
// error is read here, so that it does not turn up in the launch check of some other call.
bool wait_device(int dev)
{
    Cache &c = cache();
    std::list<Block> due, due_pinned;
    void *token = nullptr;
    int now = dev;
    cudaGetDevice(&now);
    if (now != dev) cudaSetDevice(dev);
    {
        std::lock_guard<std::mutex> lock(c.mu);
        due = take_of(c.held, dev);
        due_pinned = take_of(c.held_pinned, dev);
        std::list<void *> &tokens = c.tokens[dev];
        if (!tokens.empty()) {
            token = tokens.front();
            tokens.pop_front();
        }
        void *&anchor = c.anchor[dev];
        if (!anchor) anchor = small_block();
    }
    if (!token) token = small_block();
    // (no block to free: memory has run out, or the allocation is what a capture refuses)
    const bool ok = (token ? cudaFree(token) : cudaDeviceSynchronize()) == cudaSuccess;
    if (!ok) cudaGetLastError();
    else if (token) token = small_block();
    if (now != dev) cudaSetDevice(now);
    std::lock_guard<std::mutex> lock(c.mu);
    if (token) c.tokens[dev].push_back(token);
    if (ok) {
        for (const Block &k : due) keep_idle(c, k);
        for (const Block &k : due_pinned) keep_pinned(c, k);
    } else {
        c.held.splice(c.held.end(), due);
        c.held_pinned.splice(c.held_pinned.end(), due_pinned);
    }
    return ok;
}

// Takes a block out of the table of live ones; false if it is not there.
bool take_live(Cache &c, HostBuf &b, Block &k)
{
    auto it = c.live.find(b.p);
    b.p = nullptr;
    b.bytes = 0;
    if (it == c.live.end()) return false;
    k = it->second;
    c.live.erase(it);
    return true;
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
        if (e == cudaErrorMemoryAllocation) {   // once more without the idle blocks and the rounding up
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

xtgpu_status pool_get(void **p, size_t bytes, cudaStream_t s)
{
    cudaError_t e = cudaMallocAsync(p, bytes, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        int dev = 0;
        XTG_CUDA(cudaGetDevice(&dev));
        {
            Cache &c = cache();
            std::lock_guard<std::mutex> lock(c.mu);
            trim(c, dev, 0);
        }
        e = cudaMallocAsync(p, bytes, s);
    }
    if (e == cudaSuccess) return XTGPU_OK;
    *p = nullptr;
    return cuda_fail(e, "cudaMallocAsync", __FILE__, __LINE__);
}

void dput(HostBuf &b)
{
    if (!b.p) return;
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    Block k;
    if (take_live(c, b, k)) keep_idle(c, k);
}

void dfree(std::initializer_list<HostBuf *> bufs)
{
    bool any = false;
    for (HostBuf *b : bufs) any = any || b->p;
    if (!any) return;
    // the blocks' device, which need not be the current one
    Cache &c = cache();
    int dev = 0;
    {
        std::lock_guard<std::mutex> lock(c.mu);
        for (HostBuf *b : bufs)
            if (b->p && c.live.count(b->p)) dev = c.live[b->p].dev;
    }
    const bool waited = wait_device(dev);
    std::lock_guard<std::mutex> lock(c.mu);
    for (HostBuf *b : bufs) {
        Block k;
        if (!b->p || !take_live(c, *b, k)) continue;
        if (waited && k.dev == dev) keep_idle(c, k);
        else c.held.push_back(k);
    }
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
    } else if (cudaHostAlloc(&k.p, k.cap, cudaHostAllocPortable) != cudaSuccess) {
        // no memory to pin: the copies work on any, if slower, as they did on the caller's
        cudaGetLastError();
        k.pageable = true;
        if (!(k.p = malloc(k.cap))) {
            set_error("no host memory for staging");
            return XTGPU_ERR_NOMEM;
        }
    }
    c.live[k.p] = k;
    b.p = k.p;
    b.bytes = bytes;
    return XTGPU_OK;
}

void stage_put(HostBuf &b, bool idle)
{
    if (!b.p) return;
    int dev = 0;
    if (!idle) {
        cudaGetDevice(&dev);
        idle = wait_device(dev);
    }
    Cache &c = cache();
    std::lock_guard<std::mutex> lock(c.mu);
    Block k;
    if (!take_live(c, b, k)) return;
    if (idle) {
        keep_pinned(c, k);
    } else {
        k.dev = dev;
        c.held_pinned.push_back(k);
    }
}

// What is idle goes back to the driver: device blocks of all devices and pinned ones.
static uint64_t release_idle()
{
    Cache &c = cache();
    std::list<int> held;
    {
        std::lock_guard<std::mutex> lock(c.mu);
        for (const std::list<Block> *l : {&c.held, &c.held_pinned})
            for (const Block &k : *l) held.push_back(k.dev);
    }
    held.sort();
    held.unique();
    for (int dev : held) wait_device(dev);
    std::lock_guard<std::mutex> lock(c.mu);
    uint64_t bytes = 0;
    for (auto &kv : c.kept) {
        bytes += kv.second;
        trim(c, kv.first, 0);
        bytes -= kv.second;
    }
    while (!c.pinned.empty()) {
        if (cudaFreeHost(c.pinned.front().p) != cudaSuccess) {
            cudaGetLastError();
            break;
        }
        c.pinned_kept -= c.pinned.front().cap;
        c.pinned.pop_front();
    }
    return bytes;
}

bool host_memory(const void *p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeDevice;
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

extern "C" xtgpu_status xtgpu_release_memory(uint64_t *bytes)
{
    const uint64_t n = xtg::release_idle();
    if (bytes) *bytes = n;
    return XTGPU_OK;
}
