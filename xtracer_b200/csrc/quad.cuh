// Closest-hit traversal of the FP32 and Q8 trees.  Their nodes hold up to four
// children: the two levels below one node of the binary hierarchy, so a ray
// waits for half as many dependent node loads as on binary nodes, at the same
// number of box tests.
//
// The lanes of a warp walk together in rounds (Aila and Laine, "Understanding
// the Efficiency of Ray Traversal on GPUs", HPG 2009: speculative while-while).
// In a round every lane visits nodes until nearly all lanes hold a leaf; a lane
// that has found one puts it aside and goes on.  Then the lanes test their
// leaves together.  Node visits and primitive tests so run with most of their
// lanes instead of by turns in each step.
#pragma once

#include "traverse.cuh"

namespace xtg {

// "nothing to visit": a leaf ref of count 0 that no build produces (EMPTY_REF,
// an unused child slot, is a leaf of no primitives like any other)
constexpr int32_t DONE_REF = ~(1 << LEAF_BITS);

// A round ends when at most a quarter of the lanes with work still look for a
// leaf (then at least one of the others holds one, so every round tests one).
// us for 1 Mi bounce rays on terrain200k / terrain1m / hairball1m / spheres4096,
// FP32 trees of leaf size 2:
//   one node or leaf a step, binary nodes (before)       469 / 563 / 1025 / 97
//   rounds that wait for the last lane, binary nodes     382 / 482 /  831 / 93
//   the same on four-child nodes                         372 / 456 /  760 / 91
//   to 4 lanes (none when 8 or fewer have work)          351 / 426 /  751 / 88
//   to an eighth / to a quarter                355 / 430 / 750 / 88, 355 / 412 / 743 / 87
// Q8 501 / 601 / 1086 / 106 before, 345 / 407 / 704 / 90 now.  A batch of 60,000 such
// rays, which lasts as long as its longest walks, 150 -> 120 us on terrain200k.
constexpr int ROUND_SHARE_LOG2 = 2;

// Entry distance as an unsigned sort key with the child slot in its low bits
// (cutting them off only makes the distance smaller).  Zero stands for zero and
// all negative distances.
constexpr uint32_t MISS_KEY = 0xffffffffu;
__device__ __forceinline__ uint32_t child_key(float tn, float tf, float scale, uint32_t slot)
{
    return tn <= tf * scale ? (((uint32_t)max(__float_as_int(tn), 0) & ~3u) | slot) : MISS_KEY;
}

// The sort keys of the four children (MISS_KEY where the box is not hit) and
// their refs.  `oct` holds the signs of the ray's inverse direction: the near
// plane of an axis is the lower bound when the ray goes up that axis.
struct Quad {
    uint32_t k0, k1, k2, k3;
    int4 ref;
};

template <int FMT>
__device__ __forceinline__ void node_quad(const void *nodes, int32_t i, const RayPre &r, uint32_t oct, float tmin,
                                          float tmax, Quad &Q);

// 128-byte node: lo.x[4] hi.x[4] lo.y[4] hi.y[4] lo.z[4] hi.z[4] ref[4] -
template <>
__device__ __forceinline__ void node_quad<XTGPU_NODES_FP32>(const void *nodes, int32_t i, const RayPre &r,
                                                            uint32_t oct, float tmin, float tmax, Quad &Q)
{
    const float4 *p = (const float4 *)nodes + 8 * (size_t)i;
    const uint32_t sx = oct & 1u, sy = (oct >> 1) & 1u, sz = oct >> 2;
    const float4 nx = __ldg(p + sx), fx = __ldg(p + (sx ^ 1u));
    const float4 ny = __ldg(p + 2 + sy), fy = __ldg(p + 2 + (sy ^ 1u));
    const float4 nz = __ldg(p + 4 + sz), fz = __ldg(p + 4 + (sz ^ 1u));
    Q.ref = __ldg((const int4 *)(p + 6));
#define XTG_CHILD(c, s)                                                                                              \
    child_key(fmaxf(fmaxf(fmaf(nx.c, r.inv.x, -r.oinv.x), fmaf(ny.c, r.inv.y, -r.oinv.y)),                           \
                    fmaxf(fmaf(nz.c, r.inv.z, -r.oinv.z), tmin)),                                                    \
              fminf(fminf(fmaf(fx.c, r.inv.x, -r.oinv.x), fmaf(fy.c, r.inv.y, -r.oinv.y)),                           \
                    fminf(fmaf(fz.c, r.inv.z, -r.oinv.z), tmax)),                                                    \
              XTG_TFAR_SCALE, s)
    Q.k0 = XTG_CHILD(x, 0u);
    Q.k1 = XTG_CHILD(y, 1u);
    Q.k2 = XTG_CHILD(z, 2u);
    Q.k3 = XTG_CHILD(w, 3u);
#undef XTG_CHILD
}

// Slightly larger far-distance scale for the quantised test, whose bounds are
// formed in t-space as q * (scale * inv) + (origin * inv - o * inv).
#define XTG_TFAR_SCALE_Q8 1.0000015f

// 64-byte node: origin xyz with a biased power-of-two scale exponent in each low
// byte, -; then, one byte per child, lo.x hi.x lo.y hi.y lo.z hi.z, -, -; ref[4].
// The slab test runs in quantised space: t(q) = q * (s * inv) + (o - ray.o) * inv,
// one FMA per bound.
template <>
__device__ __forceinline__ void node_quad<XTGPU_NODES_Q8>(const void *nodes, int32_t i, const RayPre &r, uint32_t oct,
                                                          float tmin, float tmax, Quad &Q)
{
    const uint4 *p = (const uint4 *)nodes + 4 * (size_t)i;
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    const uint2 c = __ldg((const uint2 *)(p + 2));
    Q.ref = __ldg((const int4 *)(p + 3));
    const float ax = __uint_as_float((a.x & 0xFFu) << 23) * r.inv.x;
    const float ay = __uint_as_float((a.y & 0xFFu) << 23) * r.inv.y;
    const float az = __uint_as_float((a.z & 0xFFu) << 23) * r.inv.z;
    const float bx = fmaf(__uint_as_float(a.x & ~0xFFu), r.inv.x, -r.oinv.x);
    const float by = fmaf(__uint_as_float(a.y & ~0xFFu), r.inv.y, -r.oinv.y);
    const float bz = fmaf(__uint_as_float(a.z & ~0xFFu), r.inv.z, -r.oinv.z);
    const uint32_t nx = (oct & 1u) ? b.y : b.x, fx = (oct & 1u) ? b.x : b.y;
    const uint32_t ny = (oct & 2u) ? b.w : b.z, fy = (oct & 2u) ? b.z : b.w;
    const uint32_t nz = (oct & 4u) ? c.y : c.x, fz = (oct & 4u) ? c.x : c.y;
#define XTG_Q(w, k) ((float)(((w) >> (8 * (k))) & 0xFFu))
#define XTG_CHILD(k)                                                                                                 \
    child_key(fmaxf(fmaxf(fmaf(XTG_Q(nx, k), ax, bx), fmaf(XTG_Q(ny, k), ay, by)),                                   \
                    fmaxf(fmaf(XTG_Q(nz, k), az, bz), tmin)),                                                        \
              fminf(fminf(fmaf(XTG_Q(fx, k), ax, bx), fmaf(XTG_Q(fy, k), ay, by)),                                   \
                    fminf(fmaf(XTG_Q(fz, k), az, bz), tmax)),                                                        \
              XTG_TFAR_SCALE_Q8, k)
    Q.k0 = XTG_CHILD(0);
    Q.k1 = XTG_CHILD(1);
    Q.k2 = XTG_CHILD(2);
    Q.k3 = XTG_CHILD(3);
#undef XTG_CHILD
#undef XTG_Q
}

__device__ __forceinline__ void sort2(uint32_t &a, uint32_t &b)
{
    const uint32_t lo = min(a, b);
    b = max(a, b);
    a = lo;
}
__device__ __forceinline__ int32_t ref_of(const int4 &r, uint32_t key)
{
    const int32_t lo = (key & 1u) ? r.y : r.x, hi = (key & 1u) ? r.w : r.z;
    return (key & 2u) ? hi : lo;
}

// The next stack entry that may still hold a nearer hit, or one as near.
__device__ __forceinline__ int32_t pop_ref(const uint2 *stack, int &sp, float tmax)
{
    while (sp > 0) {
        const uint2 e = stack[--sp];
        if (e.y == 0u || __uint_as_float(e.y) <= tmax) return (int32_t)e.x;
    }
    return DONE_REF;
}

// Traversal state of a lane: the node or leaf it goes to next, a leaf put
// aside, and the entries of the stack (ref, entry distance).
struct QuadWalk {
    int32_t ref = DONE_REF, leaf = DONE_REF;
    int sp = 0;
    __device__ __forceinline__ void start(int32_t root)
    {
        // a scene of one leaf, or of none, has no node
        ref = root >= 0 ? root : DONE_REF;
        leaf = root >= 0 ? DONE_REF : root;
        sp = 0;
    }
    __device__ __forceinline__ bool done() const { return ref == DONE_REF && leaf == DONE_REF; }
};

// One round of the warp (all 32 lanes call it; a lane without a ray has ref and
// leaf DONE_REF).  A lane is done when both are DONE_REF again.  The stack holds
// at most three entries per level of four-child nodes.
template <int FMT, int STACK, class RAY>
__device__ __forceinline__ void quad_round(const SceneView &V, const RayPre &r, const RAY &ray, uint32_t oct, float tmin, float &tmax,
                                           uint32_t &prim, float &bu, float &bv, QuadWalk &w, uint2 *stack,
                                           int32_t *ctl_overflow, uint32_t &nv, uint32_t &np)
{
    const unsigned with = __ballot_sync(0xffffffffu, !w.done());
    const int stop = __popc(with) >> ROUND_SHARE_LOG2;
    while (true) {
        const unsigned need = __ballot_sync(0xffffffffu, w.ref >= 0 && w.leaf == DONE_REF);
        if (__popc(need) <= stop) break;
        if (w.ref >= 0) {
            Quad Q;
            node_quad<FMT>(V.nodes, w.ref, r, oct, tmin, tmax, Q);
            sort2(Q.k0, Q.k1);
            sort2(Q.k2, Q.k3);
            sort2(Q.k0, Q.k2);
            sort2(Q.k1, Q.k3);
            sort2(Q.k1, Q.k2);
            // a full stack or a walk without end (a corrupted tree): report, never loop forever
            if (w.sp > STACK - 3 || ++nv > (1u << 22)) {
                *ctl_overflow = 1;
                w.sp = 0;
                w.ref = DONE_REF;
            } else if (Q.k0 != MISS_KEY) {
                if (Q.k3 != MISS_KEY) stack[w.sp++] = make_uint2((uint32_t)ref_of(Q.ref, Q.k3), Q.k3 & ~3u);
                if (Q.k2 != MISS_KEY) stack[w.sp++] = make_uint2((uint32_t)ref_of(Q.ref, Q.k2), Q.k2 & ~3u);
                if (Q.k1 != MISS_KEY) stack[w.sp++] = make_uint2((uint32_t)ref_of(Q.ref, Q.k1), Q.k1 & ~3u);
                w.ref = ref_of(Q.ref, Q.k0);
            } else {
                w.ref = pop_ref(stack, w.sp, tmax);
            }
            if (w.ref < 0 && w.leaf == DONE_REF) {
                w.leaf = w.ref;
                if (w.ref != DONE_REF) w.ref = pop_ref(stack, w.sp, tmax);
            }
        }
    }
    if (w.leaf != DONE_REF) {
        np += leaf_count(w.leaf);
        leaf_test(V, w.leaf, ray, tmin, tmax, prim, bu, bv);
        w.leaf = DONE_REF;
        if (w.ref < 0 && w.ref != DONE_REF) {
            w.leaf = w.ref;
            w.ref = pop_ref(stack, w.sp, tmax);
        }
    }
}

}  // namespace xtg
