// 8-wide BVH with 8-bit quantised child bounds, collapsed from the binary LBVH
// on the device.  The node layout, the traversal order and the cost-optimal
// collapse follow Ylitie, Karras and Laine, "Efficient Incoherent Ray Traversal
// on GPUs Through Compressed Wide BVHs" (HPG 2017).
//
// Which binary nodes become wide nodes, and which subtrees become leaves, is
// chosen one of two ways (xtgpu_tuning::wide_collapse):
//   * 1, cost-optimal (default): a bottom-up dynamic programme over the binary
//     tree (k_wide_dp) gives every node n and budget i = 1..7 the lowest
//     surface-area cost C(n, i) of representing n's subtree by at most i
//     children of a wide node.  C(n, 1) is the cheaper of one leaf (at most 3
//     primitives: A(n) * c_prim * P(n)) and one internal wide node (A(n) *
//     c_node + the best split of 8 children between n's two binary
//     children); C(n, i > 1) is the better of C(n, i - 1) and the best split of
//     i between the two children.  The emission follows the recorded choices;
//   * 0, greedy: a wide node repeatedly opens the internal child with the
//     largest surface area until it has 8 children or only leaves are left,
//     and every binary leaf is one wide leaf.
//
// Build, one kernel launch per level of the wide tree (top down), eight lanes a node:
//   * a wide node starts from one binary internal node and takes its children
//     as above;
//   * the children take slots by direction: the child whose centroid lies
//     furthest towards octant s (relative to the node's centre) gets slot s, so
//     a ray visits slots in the order slot ^ m (m = the ray's sign bits) and
//     meets nearer children first;
//   * internal children get consecutive node indices in slot order (base + the
//     number of internal children in lower slots); the primitives of the leaf
//     children are copied next to each other (base + a 5-bit offset per child),
//     so one node names all of them.
//
// Node, 80 bytes (5 x uint4):
//   w[0..2]  origin x, y, z (float bits; the low byte holds the biased
//            power-of-two exponent of that axis' quantum)
//   w[3]     imask: bit s set if slot s is an internal child
//   w[4]     index of the first internal child
//   w[5]     index of the first leaf primitive
//   w[6..7]  meta[8]: leaf slot = (count << 5) | offset, 0 otherwise
//   w[8..19] qlo.x[8] qlo.y[8] qlo.z[8] qhi.x[8] qhi.y[8] qhi.z[8]; an unused
//            slot has qlo = 255 > qhi = 0 and is never hit
#include <algorithm>
#include <vector>

#include "xtgpu_internal.cuh"
#include "wide.cuh"

namespace xtg {

namespace {

struct WideItem {
    int32_t bref;   // binary node (>= 0) or leaf ref (< 0) the wide node starts from
    int32_t widx;   // index of the wide node
};

__device__ __forceinline__ uint32_t origin_bits_w(float v)
{
    uint32_t b = __float_as_uint(v);
    if (v == 0.f) return 0u;
    if (b & 0x80000000u) {   // negative: round the magnitude up
        uint32_t m = b & 0x7fffffffu;
        m = (m + 0xFFu) & ~0xFFu;
        return m | 0x80000000u;
    }
    return b & ~0xFFu;
}

// smallest biased exponent e (quantum 2^(e-127)) with origin + 254 quanta >= hi
__device__ __forceinline__ uint32_t pick_exp_w(float origin, float hi)
{
    float ext = hi - origin;
    uint32_t e = 1;
    if (ext > 0.f) {
        int ex;
        frexpf(ext / 255.0f, &ex);
        e = (uint32_t)max(1, min(254, ex + 127 - 1));
    }
    while (e < 254 && __fmaf_rn(254.0f, __uint_as_float(e << 23), origin) < hi) ++e;
    return e;
}

// outward-rounded quantised bounds with one quantum of padding on each side
__device__ __forceinline__ void quant_w(float lo, float hi, float o, float sc, uint32_t &qlo, uint32_t &qhi)
{
    float a = floorf(__fdiv_rd(__fsub_rd(lo, o), sc));
    float b = ceilf(__fdiv_ru(__fsub_ru(hi, o), sc));
    int ql = (int)fmaxf(0.f, fminf(255.f, a));
    int qh = (int)fmaxf(0.f, fminf(255.f, b));
    while (ql > 0 && __fmaf_rn((float)ql, sc, o) > lo) --ql;
    while (qh < 255 && __fmaf_rn((float)qh, sc, o) < hi) ++qh;
    qlo = (uint32_t)max(0, ql - 1);
    qhi = (uint32_t)min(255, qh + 1);
}

__device__ __forceinline__ float area_of(float3 lo, float3 hi)
{
    float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

// box of a leaf's primitives (the root of a scene no larger than one leaf)
__device__ void leaf_box(const float4 *prims, int32_t ref, float3 &lo, float3 &hi)
{
    lo = make_float3(INFINITY, INFINITY, INFINITY);
    hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
    uint32_t first = leaf_first(ref), cnt = leaf_count(ref);
    for (uint32_t k = 0; k < cnt; ++k) {
        const float4 *p = prims + 3 * (size_t)(first + k);
        float4 a = p[0], b = p[1], c = p[2];
        if (__float_as_uint(a.w) & SPHERE_BIT) {
            lo = make_float3(fminf(lo.x, __fsub_rd(a.x, b.x)), fminf(lo.y, __fsub_rd(a.y, b.x)),
                             fminf(lo.z, __fsub_rd(a.z, b.x)));
            hi = make_float3(fmaxf(hi.x, __fadd_ru(a.x, b.x)), fmaxf(hi.y, __fadd_ru(a.y, b.x)),
                             fmaxf(hi.z, __fadd_ru(a.z, b.x)));
        } else {
            lo = make_float3(fminf(lo.x, fminf(a.x, fminf(b.x, c.x))), fminf(lo.y, fminf(a.y, fminf(b.y, c.y))),
                             fminf(lo.z, fminf(a.z, fminf(b.z, c.z))));
            hi = make_float3(fmaxf(hi.x, fmaxf(a.x, fmaxf(b.x, c.x))), fmaxf(hi.y, fmaxf(a.y, fmaxf(b.y, c.y))),
                             fmaxf(hi.z, fmaxf(a.z, fmaxf(b.z, c.z))));
        }
    }
}

// child c (0 or 1) of binary node i: its ref and box
__device__ __forceinline__ void bin_child(const float4 *nodes, int32_t i, int c, int32_t &ref, float3 &lo, float3 &hi)
{
    const float4 *p = nodes + 4 * (size_t)i;
    float4 a = p[c], z = p[2], d = p[3];
    lo = make_float3(a.x, a.z, c == 0 ? z.x : z.z);
    hi = make_float3(a.y, a.w, c == 0 ? z.y : z.w);
    ref = __float_as_int(c == 0 ? d.x : d.y);
}

// --- cost-optimal collapse --------------------------------------------------
// Per binary internal node: C(n, i) for i = 1..7, the left child's share k of
// the best split of j = 2..8 children, which C(n, i) come from a split (bit
// i - 1, i >= 2) and whether C(n, 1) is a leaf (bit 7), and P(n).
struct WideDP {
    float c[7];
    uint8_t split[7];
    uint8_t use;
    int32_t prims;
};

constexpr float WIDE_NODE_COST = 1.0f;

__device__ __forceinline__ float3 fmin3(float3 a, float3 b)
{
    return make_float3(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z));
}
__device__ __forceinline__ float3 fmax3(float3 a, float3 b)
{
    return make_float3(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z));
}

__global__ void k_wide_parents(int ni, const float4 *__restrict__ bnodes, int32_t *__restrict__ parent)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ni) return;
    const float4 d = bnodes[4 * (size_t)n + 3];
    const int32_t c0 = __float_as_int(d.x), c1 = __float_as_int(d.y);
    if (c0 >= 0 && c0 < ni) parent[c0] = n;
    if (c1 >= 0 && c1 < ni) parent[c1] = n;
}

// the DP entry of binary node n from its children's (computed before)
__device__ void wide_dp_node(const float4 *__restrict__ bnodes, WideDP *dp, int32_t n, float cprim)
{
    float ck[2][7];
    int32_t pk[2];
    float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
    for (int c = 0; c < 2; ++c) {
        int32_t ref;
        float3 cl, ch;
        bin_child(bnodes, n, c, ref, cl, ch);
        lo = fmin3(lo, cl);
        hi = fmax3(hi, ch);
        if (ref >= 0) {
            // written by another thread before its fence: read past L1
            const float *src = (const float *)(dp + ref);
            for (int i = 0; i < 7; ++i) ck[c][i] = __ldcg(src + i);
            pk[c] = __ldcg(&dp[ref].prims);
        } else {
            const int cnt = (int)leaf_count(ref);
            const float v = ref == EMPTY_REF ? 0.f : area_of(cl, ch) * cprim * (float)cnt;
            for (int i = 0; i < 7; ++i) ck[c][i] = v;
            pk[c] = cnt;
        }
    }
    WideDP out;
    out.prims = pk[0] + pk[1];
    float dist[9];
    for (int j = 2; j <= 8; ++j) {
        float best = INFINITY;
        int bk = 1;
        for (int k = 1; k < j; ++k) {
            const float v = ck[0][k - 1] + ck[1][j - k - 1];
            if (v < best) {
                best = v;
                bk = k;
            }
        }
        dist[j] = best;
        out.split[j - 2] = (uint8_t)bk;
    }
    const float A = area_of(lo, hi);
    const float cleaf = out.prims <= WIDE_MAX_LEAF ? A * cprim * (float)out.prims : INFINITY;
    const float cint = A * WIDE_NODE_COST + dist[8];
    out.use = 0;
    out.c[0] = fminf(cleaf, cint);
    if (cleaf <= cint) out.use |= 0x80u;
    for (int i = 2; i <= 7; ++i) {
        if (dist[i] < out.c[i - 2]) {
            out.c[i - 1] = dist[i];
            out.use |= (uint8_t)(1u << (i - 1));
        } else {
            out.c[i - 1] = out.c[i - 2];
        }
    }
    dp[n] = out;
}

// Bottom up: a thread starts at every node without internal children and
// climbs while it is the last of a node's internal children to finish.
__global__ void k_wide_dp(int ni, const float4 *__restrict__ bnodes, const int32_t *__restrict__ parent,
                          unsigned *__restrict__ arrived, WideDP *dp, float cprim, int *err)
{
    int32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= ni) return;
    {
        const float4 d = bnodes[4 * (size_t)n + 3];
        if (__float_as_int(d.x) >= 0 || __float_as_int(d.y) >= 0) return;
    }
    for (int guard = 0;; ++guard) {
        if (guard > 256) {   // deeper than any tree this build makes: report, never loop forever
            atomicExch(err, 1);
            return;
        }
        wide_dp_node(bnodes, dp, n, cprim);
        __threadfence();
        const int32_t p = parent[n];
        if (p < 0) return;
        const float4 d = bnodes[4 * (size_t)p + 3];
        const unsigned need = (__float_as_int(d.x) >= 0 ? 1u : 0u) + (__float_as_int(d.y) >= 0 ? 1u : 0u);
        if (atomicAdd(&arrived[p], 1u) + 1u < need) return;
        __threadfence();
        n = p;
    }
}

// Eight lanes make one wide node, a lane a child slot of its list of children (a
// thread a node spent 4000 instructions on placing them, one after another, so each
// of the tree's ten or so levels lasted as long as one node: 609 us for the 11
// levels of a 500k-triangle terrain).
constexpr int WIDE_BLOCK = 128;

// Or, sum, minimum and maximum over the eight lanes of a node.
template <class T, class F>
__device__ __forceinline__ T reduce8(T v, F f)
{
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, o, 8));
    return v;
}
__device__ __forceinline__ float min8(float v) { return reduce8(v, [](float a, float b) { return fminf(a, b); }); }
__device__ __forceinline__ float max8(float v) { return reduce8(v, [](float a, float b) { return fmaxf(a, b); }); }
__device__ __forceinline__ uint32_t or8(uint32_t v) { return reduce8(v, [](uint32_t a, uint32_t b) { return a | b; }); }
__device__ __forceinline__ int sum8(int v) { return reduce8(v, [](int a, int b) { return a + b; }); }

// The child of lane k of the wide node made from binary node `root` under the DP's
// choices, or false if it has fewer.  A subtree with a budget of i children has i
// lanes; each lane walks down to its own child, the left part's lanes first, and the
// first lane of the range has it.  A subtree chosen as a leaf becomes the leaf ref of
// its primitives (contiguous in the leaf order).
__device__ __forceinline__ bool wide_child_dp(const float4 *__restrict__ bnodes, const WideDP *__restrict__ dp,
                                              int32_t root, int k, int32_t &cref, float3 &lo, float3 &hi)
{
    int32_t ref = root;
    int first = 0, i = 8;
    for (int g = 0; g < 16; ++g) {   // at most 7 splits
        int left = dp[ref].split[i - 2];
        const int side = k - first < left ? 0 : 1;
        const int32_t from = ref;
        bin_child(bnodes, from, side, ref, lo, hi);
        if (side) {
            first += left;
            i -= left;
        } else {
            i = left;
        }
        if (ref < 0) break;
        while (i > 1 && !(dp[ref].use & (1u << (i - 1)))) --i;
        if (k - first >= i) return false;   // the subtree takes fewer than its share
        if (i == 1) break;
    }
    if (k != first) return false;
    cref = ref;
    if (ref >= 0 && (dp[ref].use & 0x80u)) {
        int32_t r = ref;
        for (int g = 0; r >= 0 && g < 64; ++g) r = __float_as_int(bnodes[4 * (size_t)r + 3].x);
        // the subtree's primitives start at its leftmost leaf; a walk that ends on no
        // leaf (a malformed tree) keeps the node internal
        if (r < 0 && r != EMPTY_REF) cref = leaf_ref(leaf_first(r), (uint32_t)dp[ref].prims);
    }
    return true;
}

// The same without costs: the largest internal child is opened until there are 8
// children or only leaves.
__device__ __forceinline__ bool wide_child_greedy(const float4 *__restrict__ bnodes, int32_t root, int k, int32_t &cref,
                                                  float3 &lo, float3 &hi)
{
    if (k < 2) bin_child(bnodes, root, k, cref, lo, hi);
    int n = 2;
    for (int round = 0; round < 6; ++round) {   // all nodes of a warp take every round
        const float a = k < n && cref >= 0 ? area_of(lo, hi) : -1.f;
        const float ba = max8(a);
        // the first lane of that area
        const unsigned m = __ballot_sync(0xffffffffu, a == ba) >> (threadIdx.x & 24u) & 0xFFu;
        const int best = m ? __ffs(m) - 1 : 0;
        const int32_t from = __shfl_sync(0xffffffffu, cref, best, 8);
        if (!(ba >= 0.f)) continue;
        if (k == best) bin_child(bnodes, from, 0, cref, lo, hi);
        if (k == n) bin_child(bnodes, from, 1, cref, lo, hi);
        ++n;
    }
    return k < n;
}

// ctr: [0] wide nodes allocated, [1] leaf primitives placed, [2] error flag, and from
// [4] the number of nodes of each level.  The level's count is read from memory, so
// the levels are launched one after another without asking how many there are
// (wide_level_nodes: none once the flag is set).
__global__ void __launch_bounds__(WIDE_BLOCK)
    k_wide_level(const float4 *__restrict__ bnodes, const float4 *__restrict__ bprims, const WideDP *__restrict__ dp,
                 const WideItem *__restrict__ items, WideItem *__restrict__ next, int level, int max_nodes,
                 uint4 *__restrict__ wnodes, float4 *__restrict__ wprims, int n_prims, int *ctr)
{
    __shared__ uint32_t node[WIDE_BLOCK / 8][20];
    __shared__ int count;
    if (threadIdx.x == 0) count = wide_level_nodes(ctr, level, max_nodes);
    __syncthreads();
    const int nitems = count;
    const int k = threadIdx.x & 7, g = threadIdx.x >> 3;
    uint32_t *W = node[g];
    uint8_t *B = (uint8_t *)W;
    for (int base = blockIdx.x * (WIDE_BLOCK / 8); base < nitems; base += gridDim.x * (WIDE_BLOCK / 8)) {
        const int it = base + g;
        const bool on = it < nitems;   // the block's lanes stay together
        const WideItem I = on ? items[it] : WideItem{0, 0};
        int32_t cref = EMPTY_REF;
        float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
        bool have = false;
        if (!dp) {
            // (the lanes of nodes that start from a leaf or are off go along on node 0)
            have = wide_child_greedy(bnodes, on && I.bref >= 0 ? I.bref : 0, k, cref, lo, hi) && on && I.bref >= 0;
        } else if (on && I.bref >= 0) {
            have = wide_child_dp(bnodes, dp, I.bref, k, cref, lo, hi);
        }
        if (on && I.bref < 0 && k == 0) {
            cref = I.bref;
            leaf_box(bprims, I.bref, lo, hi);
            have = true;
        }
        have = have && cref != EMPTY_REF;   // empty leaves are dropped
        if (!have) {
            lo = make_float3(INFINITY, INFINITY, INFINITY);
            hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
        }
        // node box and centre
        float3 nlo = make_float3(min8(lo.x), min8(lo.y), min8(lo.z)), nhi = make_float3(max8(hi.x), max8(hi.y), max8(hi.z));
        const int n = __popc(__ballot_sync(0xffffffffu, have) >> (threadIdx.x & 24u) & 0xFFu);
        if (n == 0) nlo = nhi = make_float3(0.f, 0.f, 0.f);
        const float3 c = make_float3(0.5f * (lo.x + hi.x) - 0.5f * (nlo.x + nhi.x), 0.5f * (lo.y + hi.y) - 0.5f * (nlo.y + nhi.y),
                                     0.5f * (lo.z + hi.z) - 0.5f * (nlo.z + nhi.z));
        // slots: greedily the (child, slot) pair whose centroid lies furthest towards
        // the slot's octant, the first child and its lowest slot among equals
        int slot = -1;
        uint32_t taken = 0;
        for (int round = 0; round < 8; ++round) {
            float bv = -INFINITY;
            int bs = -1;
            if (have && slot < 0)
                for (int s = 0; s < 8; ++s) {
                    const float v = ((s & 1) ? c.x : -c.x) + ((s & 2) ? c.y : -c.y) + ((s & 4) ? c.z : -c.z);
                    if (!(taken & (1u << s)) && (bs < 0 || v > bv)) {
                        bv = v;
                        bs = s;
                    }
                }
            const float best = max8(bv);
            // (a child whose distances are not numbers still takes a slot)
            const unsigned cand = __ballot_sync(0xffffffffu, bs >= 0 && !(bv < best)) >> (threadIdx.x & 24u) & 0xFFu;
            const int win = cand ? __ffs(cand) - 1 : 0;
            const int ws = __shfl_sync(0xffffffffu, bs, win, 8);
            if (cand) taken |= 1u << ws;
            if (cand && k == win) slot = ws;
        }
        // internal children get nodes and leaf children places for their primitives,
        // both in slot order
        const bool internal = have && cref >= 0;
        const uint32_t imask = or8(internal ? 1u << slot : 0u);
        const int cnt = have && !internal ? (int)leaf_count(cref) : 0;
        const int ni = __popc(imask), np = sum8(cnt);
        int off = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int sj = __shfl_sync(0xffffffffu, slot, j, 8), cj = __shfl_sync(0xffffffffu, cnt, j, 8);
            if (cj && sj < slot) off += cj;
        }
        int child_base = 0, prim_base = 0, next_base = 0;
        if (k == 0) {
            if (ni) child_base = atomicAdd(&ctr[0], ni);
            if (np) prim_base = atomicAdd(&ctr[1], np);
            if (ni) next_base = atomicAdd(&ctr[4 + level + 1], ni);
        }
        child_base = __shfl_sync(0xffffffffu, child_base, 0, 8);
        prim_base = __shfl_sync(0xffffffffu, prim_base, 0, 8);
        next_base = __shfl_sync(0xffffffffu, next_base, 0, 8);
        // cannot happen for a valid binary tree; nothing of the node is written then
        const bool bad = child_base + ni > max_nodes || prim_base + np > n_prims || next_base + ni > max_nodes;
        if (bad && k == 0) atomicExch(&ctr[WIDE_CTR_ERROR], 1);
        // node: unused slots have qlo = 255 > qhi = 0
        const float alo[3] = {nlo.x, nlo.y, nlo.z}, ahi[3] = {nhi.x, nhi.y, nhi.z};
        const float cl[3] = {lo.x, lo.y, lo.z}, ch[3] = {hi.x, hi.y, hi.z};
        W[k] = 0u;
        if (k < 6) {
            W[8 + k] = 0xffffffffu;
            W[14 + k] = 0u;
        }
        __syncwarp();
        for (int x = 0; x < 3; ++x) {
            const uint32_t ob = origin_bits_w(alo[x]);
            const float o = __uint_as_float(ob);
            const uint32_t ex = pick_exp_w(o, ahi[x]);
            if (k == 0) W[x] = ob | ex;
            if (have) {
                uint32_t ql, qh;
                quant_w(cl[x], ch[x], o, __uint_as_float(ex << 23), ql, qh);
                B[32 + 8 * x + slot] = (uint8_t)ql;
                B[56 + 8 * x + slot] = (uint8_t)qh;
            }
        }
        if (k == 0) {
            W[3] = imask;
            W[4] = (uint32_t)child_base;
            W[5] = (uint32_t)prim_base;
        }
        if (cnt) B[24 + slot] = (uint8_t)((cnt << 5) | off);
        __syncwarp();
        if (on && !bad) {
            if (k < 5) wnodes[5 * (size_t)I.widx + k] = make_uint4(W[4 * k], W[4 * k + 1], W[4 * k + 2], W[4 * k + 3]);
            if (internal) {
                const int rank = __popc(imask & ((1u << slot) - 1u));
                next[next_base + rank] = WideItem{cref, child_base + rank};
            } else if (cnt) {
                const float4 *src = bprims + 3 * (size_t)leaf_first(cref);
                float4 *dst = wprims + 3 * (size_t)(prim_base + off);
                for (int j = 0; j < 3 * cnt; ++j) dst[j] = src[j];
            }
        }
        __syncwarp();
    }
}

}  // namespace

xtgpu_status build_wide(xtgpu_scene *sc, cudaStream_t s)
{
    DevScene &S = sc->dev;
    const int n = (int)sc->n_prims;
    if (sc->leaf_size > WIDE_MAX_LEAF) {
        set_error("xtgpu_bvh_build: the 8-wide format takes leaves of at most 3 primitives");
        return XTGPU_ERR_INVALID;
    }
    dfree({&sc->nodesW, &sc->leafW});
    sc->builtW = false;
    sc->depthW = 0;
    sc->n_wide = 0;
    if (n == 0) {
        S.nodesW = nullptr;
        S.leafW = nullptr;
        S.rootW = -1;
        sc->builtW = true;
        return XTGPU_OK;
    }
    // every wide node starts from a distinct binary internal node (or the root leaf)
    const int max_nodes = std::max(1, n - 1);
    XTG_TRY(dalloc(sc->nodesW, sizeof(uint4) * 5 * (size_t)max_nodes, s));
    XTG_TRY(dalloc(sc->leafW, sizeof(float4) * 3 * (size_t)n, s));
    const xtgpu_tuning &T = scene_tuning(sc);
    const int ni = n - 1;
    Scratch dp_;
    HostBuf &dpb = dp_.b;
    if (T.wide_collapse == 1 && ni > 0 && S.root >= 0) {
        // the cost tables, bottom up
        Scratch par_, arr_, err_;
        HostBuf &parb = par_.b, &arrb = arr_.b, &errb = err_.b;
        XTG_TRY(dalloc(dpb, sizeof(WideDP) * (size_t)ni, s));
        XTG_TRY(dalloc(parb, sizeof(int32_t) * (size_t)ni, s));
        XTG_TRY(dalloc(arrb, sizeof(unsigned) * (size_t)ni, s));
        XTG_TRY(dalloc(errb, sizeof(int), s));
        XTG_CUDA(cudaMemsetAsync(parb.p, 0xff, sizeof(int32_t) * (size_t)ni, s));
        XTG_CUDA(cudaMemsetAsync(arrb.p, 0, sizeof(unsigned) * (size_t)ni, s));
        XTG_CUDA(cudaMemsetAsync(errb.p, 0, sizeof(int), s));
        k_wide_parents<<<(ni + 255) / 256, 256, 0, s>>>(ni, S.nodes32, (int32_t *)parb.p);
        const float cprim = T.wide_prim_cost > 0.f ? T.wide_prim_cost : 1.0f;
        k_wide_dp<<<(ni + 127) / 128, 128, 0, s>>>(ni, S.nodes32, (const int32_t *)parb.p, (unsigned *)arrb.p,
                                                   (WideDP *)dpb.p, cprim, (int *)errb.p);
        int err = 0;
        cudaError_t e = cudaMemcpyAsync(&err, errb.p, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        par_.idle = arr_.idle = err_.idle = e == cudaSuccess;
        if (e != cudaSuccess) return cuda_fail(e, "wide collapse costs", __FILE__, __LINE__);
        if (err) {
            set_error("xtgpu_bvh_build: wide collapse costs did not reach the root");
            return XTGPU_ERR_CUDA;
        }
    }
    Scratch items_a, items_b, ctr_;
    HostBuf &itemsA = items_a.b, &itemsB = items_b.b, &ctrb = ctr_.b;
    constexpr int MAX_LEVELS = 128;   // a binary tree of depth <= 64 cannot give more levels
    constexpr int CTRS = 4 + MAX_LEVELS + 1;
    XTG_TRY(dalloc(itemsA, sizeof(WideItem) * (size_t)max_nodes, s));
    XTG_TRY(dalloc(itemsB, sizeof(WideItem) * (size_t)max_nodes, s));
    XTG_TRY(dalloc(ctrb, sizeof(int) * CTRS, s));
    int *ctr = (int *)ctrb.p;
    WideItem root{S.root, 0};
    int hctr[CTRS] = {1, 0, 0, 0, 1};
    XTG_CUDA(cudaMemcpyAsync(itemsA.p, &root, sizeof(root), cudaMemcpyHostToDevice, s));
    XTG_CUDA(cudaMemcpyAsync(ctr, hctr, sizeof(hctr), cudaMemcpyHostToDevice, s));
    WideItem *cur = (WideItem *)itemsA.p, *nxt = (WideItem *)itemsB.p;
    int levels = 0;
    xtgpu_status st = XTGPU_OK;
    // a dozen levels (an empty one costs 2 us), then a look at how far they went
    const int blocks_max = 148 * 16, per_block = WIDE_BLOCK / 8;
    for (bool more = true; more;) {
        if (levels >= MAX_LEVELS) {
            set_error("xtgpu_bvh_build: wide collapse did not terminate");
            st = XTGPU_ERR_CUDA;
            break;
        }
        for (int k = 0; k < 12 && levels < MAX_LEVELS; ++k, ++levels) {
            // level l has at most 8^l nodes
            const int64_t most = levels < 9 ? std::min<int64_t>(max_nodes, 1ll << (3 * levels)) : max_nodes;
            const int nb = (int)std::min<int64_t>((most + per_block - 1) / per_block, blocks_max);
            k_wide_level<<<nb, WIDE_BLOCK, 0, s>>>(S.nodes32, S.leaf_prims, (const WideDP *)dpb.p, cur, nxt, levels,
                                                   max_nodes, (uint4 *)sc->nodesW.p, (float4 *)sc->leafW.p, n, ctr);
            std::swap(cur, nxt);
        }
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(hctr, ctr, sizeof(hctr), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            st = cuda_fail(e, "wide collapse", __FILE__, __LINE__);
            break;
        }
        if (hctr[WIDE_CTR_ERROR]) {
            set_error("xtgpu_bvh_build: wide collapse overflow");
            st = XTGPU_ERR_CUDA;
            break;
        }
        more = hctr[4 + levels] > 0;
    }
    while (levels > 1 && hctr[4 + levels - 1] == 0) --levels;
    sc->n_wide = hctr[0];
    // every level has been waited for
    items_a.idle = items_b.idle = ctr_.idle = dp_.idle = st == XTGPU_OK;
    if (st != XTGPU_OK) {
        dfree({&sc->nodesW, &sc->leafW});
        return st;
    }
    sc->depthW = levels;
    sc->wide_collapse = T.wide_collapse;
    sc->wide_prim_cost = T.wide_prim_cost;
    S.nodesW = (const uint4 *)sc->nodesW.p;
    S.leafW = (const float4 *)sc->leafW.p;
    S.rootW = 0;
    sc->builtW = true;
    return XTGPU_OK;
}

}  // namespace xtg
