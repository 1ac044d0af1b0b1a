// Closest-hit traversal of the 8-wide quantised BVH built by wide.cu.
//
// A node visit tests its 8 child boxes in quantised space (one FMA per bound:
// t(q) = q * (2^e * inv) + (origin - ray.o) * inv), puts the primitives of
// every hit leaf child aside, and goes on with the nearest hit internal
// child.  The other hit internal children stay behind as one stack entry (node
// group): the base index, the node's internal-child mask and the hit children
// as bits in visiting order.  Visiting order is slot ^ m, m the ray's sign
// bits, which takes the children on the ray's entry side first (the build
// puts children in slots by direction).  Ylitie, Karras and Laine, HPG 2017.
#pragma once

#include "traverse.cuh"

namespace xtg {

constexpr int WIDE_MAX_LEAF = 3;

// Nodes of a level of the collapse that the level's launch may read (wide.cu, counters of
// k_wide_level).  A node that finds no room sets the flag after it has raised the next
// level's count, and writes none of its children: what the count then promises beyond the
// written ones must not be read, and the host looks only after a dozen levels.
constexpr int WIDE_CTR_ERROR = 2, WIDE_CTR_LEVEL = 4;
__host__ __device__ inline int wide_level_nodes(const int *ctr, int level, int max_nodes)
{
    const int n = ctr[WIDE_CTR_LEVEL + level];
    return ctr[WIDE_CTR_ERROR] || n < 0 || n > max_nodes ? 0 : n;
}

// far-distance scale of the quantised box test (as for the binary Q8 nodes)
#define XTG_TFAR_SCALE_W8 1.0000015f

__device__ __forceinline__ float q8(uint32_t w, int k) { return (float)((w >> (8 * k)) & 0xFFu); }

// A quantised bound as the float 1 + q / 32768, by one byte permute (byte k of the word
// into the mantissa of one) instead of an integer conversion.  Conversions run on the
// XU pipe, which 48 of them a node kept 62 % busy on the hairball, the most of any
// pipe; all of them as permutes overload the ALU instead (46 % busy, half rate) and are
// 3-8 % slower.  One axis of three balances the two: 579 -> 538 us for 1 Mi bounce rays
// on hairball1m, 372 -> 362 on terrain1m (two axes: 555, 370).
__device__ __forceinline__ float q8_biased(uint32_t w, int k)
{
    return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | (uint32_t)(k << 4)));
}

// The plane distances t(q) = q * s + b of that axis, s the quantum and b the node's
// origin in ray distance, as one FMA on q8_biased(q): (1 + q / 32768) * S + (b - S),
// S = 32768 s.  Rounding b - S moves a plane by at most half an ulp of |b| + |S|, up to
// 1/512 quantum, and adding the slack by as much again.  So near planes get their base
// two such ulps lower and far planes two higher: no box that t(q) hits is missed, and
// where the products overflow the comparisons drop the NaN and take the box.
struct BiasedAxis {
    float S, near, far;
};
__device__ __forceinline__ BiasedAxis biased_axis(uint32_t word, float inv, float oinv)
{
    BiasedAxis a;
    const float b = fmaf(__uint_as_float(word & ~0xFFu), inv, -oinv);
    a.S = __uint_as_float((word & 0xFFu) << 23) * (inv * 32768.0f);
    const float base = b - a.S, slack = fabsf(b) + fabsf(a.S);
    a.near = fmaf(slack, -0x1p-22f, base);
    a.far = fmaf(slack, 0x1p-22f, base);
    return a;
}

// Ray sign bits: bit k set if component k of the (clamped) inverse direction
// is negative; a zero component counts by the sign of its clamped inverse.
__device__ __forceinline__ uint32_t ray_octant(const RayPre &r)
{
    return (r.inv.x < 0.f ? 1u : 0u) | (r.inv.y < 0.f ? 2u : 0u) | (r.inv.z < 0.f ? 4u : 0u);
}

// Bit s of x moved to bit s ^ m (8 bits).
__device__ __forceinline__ uint32_t permute_xor8(uint32_t x, uint32_t m)
{
    if (m & 1u) x = ((x & 0x55u) << 1) | ((x >> 1) & 0x55u);
    if (m & 2u) x = ((x & 0x33u) << 2) | ((x >> 2) & 0x33u);
    if (m & 4u) x = ((x & 0x0Fu) << 4) | ((x >> 4) & 0x0Fu);
    return x;
}

// Visits `node`: the primitives of its hit leaf children as bits from `pbase` on, and
// in `node` the next node to visit, or -1 when nothing is left on the stack or it
// overflowed.
template <int STACK>
__device__ __forceinline__ void wide_visit(const SceneView &V, const RayPre &r, uint32_t m, float tmin, float tmax,
                                           int32_t &node, int &sp, uint2 *stack, int32_t *ctl_overflow,
                                           uint32_t &leaves, uint32_t &pbase)
{
    const uint4 *p = (const uint4 *)V.nodes + 5 * (size_t)node;
    const uint4 w0 = __ldg(p), w1 = __ldg(p + 1);
    // the stack's top entry, read with the node so that a pop at the end of
    // the visit does not wait for local memory (entry 0, unused, when empty)
    const uint2 top = stack[sp > 0 ? sp - 1 : 0];
    const float sx = __uint_as_float((w0.x & 0xFFu) << 23) * r.inv.x;
    const float sy = __uint_as_float((w0.y & 0xFFu) << 23) * r.inv.y;
    const float bx = fmaf(__uint_as_float(w0.x & ~0xFFu), r.inv.x, -r.oinv.x);
    const float by = fmaf(__uint_as_float(w0.y & ~0xFFu), r.inv.y, -r.oinv.y);
    const BiasedAxis az = biased_axis(w0.z, r.inv.z, r.oinv.z);
    const uint32_t imask = w0.w;
    // bound words, 4 slots each: qlo.x at word 8+h, qlo.y 10+h, qlo.z 12+h,
    // qhi.x 14+h, qhi.y 16+h, qhi.z 18+h (h = 0 for slots 0-3, 1 for 4-7).
    // Both halves unrolled, so the second half's loads are issued with the
    // first's instead of after it (a few spilled words, cheaper than the
    // second wait).  The near plane of an axis is its lower bound when the ray
    // goes up that axis, else the upper one, so each bound takes one FMA and
    // no swap.  An unused slot (qlo 255 > qhi 0) is behind its own far plane
    // and never hits.
    const uint32_t *qw = (const uint32_t *)(p + 2);
    uint32_t hitbits = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t lx = __ldg(qw + h), ly = __ldg(qw + 2 + h), lz = __ldg(qw + 4 + h);
        const uint32_t hx = __ldg(qw + 6 + h), hy = __ldg(qw + 8 + h), hz = __ldg(qw + 10 + h);
        const uint32_t nx = (m & 1u) ? hx : lx, fx = (m & 1u) ? lx : hx;
        const uint32_t ny = (m & 2u) ? hy : ly, fy = (m & 2u) ? ly : hy;
        const uint32_t nz = (m & 4u) ? hz : lz, fz = (m & 4u) ? lz : hz;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float tn = fmaxf(fmaxf(fmaf(q8(nx, k), sx, bx), fmaf(q8(ny, k), sy, by)),
                                   fmaxf(fmaf(q8_biased(nz, k), az.S, az.near), tmin));
            const float tf = fminf(fminf(fmaf(q8(fx, k), sx, bx), fmaf(q8(fy, k), sy, by)),
                                   fminf(fmaf(q8_biased(fz, k), az.S, az.far), tmax));
            hitbits |= (tn <= tf * XTG_TFAR_SCALE_W8 ? 1u : 0u) << (4 * h + k);
        }
    }
    uint32_t hits = permute_xor8(hitbits & imask, m);
    leaves = 0;
    for (uint32_t lh = hitbits & ~imask; lh; lh &= lh - 1u) {
        const int slot = __ffs(lh) - 1;
        const uint32_t mb = ((slot < 4 ? w1.z : w1.w) >> (8 * (slot & 3))) & 0xFFu;
        leaves |= ((1u << (mb >> 5)) - 1u) << (mb & 31u);
    }
    pbase = w1.y;
    uint32_t base = w1.x, im = imask;
    if (!hits) {
        // next node group from the stack
        if (sp == 0) {
            node = -1;
            return;
        }
        --sp;
        const uint2 e = top;
        base = e.x;
        im = e.y & 0xFFu;
        hits = e.y >> 8;
    }
    const int key = __ffs(hits) - 1;
    hits &= hits - 1u;
    const uint32_t slot = (uint32_t)key ^ m;
    node = (int32_t)(base + (uint32_t)__popc(im & ((1u << slot) - 1u)));
    if (hits) {
        if (sp >= STACK) {
            *ctl_overflow = 1;
            node = -1;
            return;
        }
        stack[sp++] = make_uint2(base, im | (hits << 8));
    }
}

// Traversal state of a lane: the node to visit next (-1: none), the stack's entries,
// and the primitives of up to two visited nodes that wait for their tests.
struct WideWalk {
    int32_t ref = -1;
    int sp = 0;
    uint32_t la = 0, pa = 0, lb = 0, pb = 0;
    __device__ __forceinline__ void start(int32_t root)   // -1 for an empty tree
    {
        ref = root;
        sp = 0;
        la = lb = 0u;
    }
    __device__ __forceinline__ bool done() const { return ref < 0 && !la; }
};

// A round ends when at most this share (of 32) of the lanes with work have no
// primitives to test.  One node visit and its primitives a step ran the tests with 2.6
// of 32 lanes, and up to 2.3 of their loops a step.  us for 1 Mi bounce rays on
// terrain200k / terrain1m / hairball1m / phong160k / spheres64:
//   a step each (before)   374 / 433 / 603 / 299 / 64
//   share 1                386 / 444 / 704 / 335 / 60
//   share 8                342 / 391 / 605 / 281 / 57
//   share 12 / 14          323 / 371 / 576 / 271 / 56, 325 / 371 / 561 / 270 / 55
//   share 20               350 / 405 / 591 / 293 / 57
// Waiting longer visits more nodes with a stale closest hit (hairball 16.5 a ray
// before, 16.9 at 14, 17.6 at 1).
constexpr int WIDE_ROUND_SHARE = 14;

// One round of the warp (all 32 lanes call it): every lane visits nodes, puts the
// primitives that it meets aside and goes on until it meets a second set; then the
// lanes test one set each together (speculative while-while, as quad_round).
template <int STACK, class RAY>
__device__ __forceinline__ void wide_round(const SceneView &V, const RayPre &r, const RAY &ray, uint32_t m, float tmin, float &tmax,
                                           uint32_t &prim, float &bu, float &bv, WideWalk &w, uint2 *stack,
                                           int32_t *ctl_overflow, uint32_t &nv, uint32_t &np)
{
    const unsigned with = __ballot_sync(0xffffffffu, !w.done());
    const int stop = (__popc(with) * WIDE_ROUND_SHARE) >> 5;
    while (true) {
        const unsigned need = __ballot_sync(0xffffffffu, w.ref >= 0 && !w.la);
        if (__popc(need) <= stop) break;
        if (w.ref >= 0 && !w.lb) {
            uint32_t l, p;
            wide_visit<STACK>(V, r, m, tmin, tmax, w.ref, w.sp, stack, ctl_overflow, l, p);
            if (++nv > (1u << 22)) {   // corrupted tree: report, never loop forever
                *ctl_overflow = 1;
                w.ref = -1;
            }
            if (l && !w.la) {
                w.la = l;
                w.pa = p;
            } else if (l) {
                w.lb = l;
                w.pb = p;
            }
        }
    }
    while (w.la) {
        const int k = __ffs(w.la) - 1;
        w.la &= w.la - 1u;
        ++np;
        prim_test(V.leaf, w.pa + (uint32_t)k, ray, tmin, tmax, prim, bu, bv);
    }
    w.la = w.lb;
    w.pa = w.pb;
    w.lb = 0u;
}

// Closest hit of one ray, each node's primitives tested at once.
template <int STACK>
__device__ __forceinline__ void trace_wide(const SceneView &V, const RayPre &r, float tmin, float &tmax,
                                           uint32_t &prim, float &bu, float &bv, int32_t *ctl_overflow, uint32_t &nv,
                                           uint32_t &np)
{
    const uint32_t m = ray_octant(r);
    uint2 stack[STACK];
    stack[0] = make_uint2(0u, 0u);   // wide_visit reads entry 0 ahead even when the stack is empty
    int sp = 0;
    for (int32_t node = V.root; node >= 0;) {
        uint32_t leaves, base;
        wide_visit<STACK>(V, r, m, tmin, tmax, node, sp, stack, ctl_overflow, leaves, base);
        while (leaves) {
            const int k = __ffs(leaves) - 1;
            leaves &= leaves - 1u;
            ++np;
            prim_test(V.leaf, base + (uint32_t)k, RegRay{r}, tmin, tmax, prim, bu, bv);
        }
        if (++nv > (1u << 22)) {   // corrupted tree: report, never loop forever
            *ctl_overflow = 1;
            break;
        }
    }
    for (int p = 0; p < V.n_planes; ++p)
        if (hit_plane(r, __ldg(V.planes + p), tmin, tmax)) {
            prim = V.plane_base + (uint32_t)p;
            bu = bv = 0.f;
        }
}

}  // namespace xtg
