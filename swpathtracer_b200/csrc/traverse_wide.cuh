// traverse_wide.cuh -- closest hit over the 8-wide quantized BVH (wide_build.h).
//
// Why the answer is still the reference's: every box of the reference tree below the root is its
// primitives' bounds inflated by 1e-3 (acceleration/sbvh.cpp:409-412), and the wide nodes' boxes
// contain those boxes (quantized outward).  A hit the reference keeps lies inside its leaf box
// (inside() below), hence at least ~1e-3 inside every ancestor box, so a conservative box test --
// here one FMA per plane on the quantized grid, with the interval clipped to [0, best t] -- can only
// visit more nodes than needed, never skip the node holding that hit.  The root box is tested with the
// reference's own slab test first, and every candidate is accepted by the reference's exact rules:
// Moller-Trumbore as in triangle.cpp, t > 0, the hit point inside the reference leaf box (+-1e-3), and
// the smallest (t, rank) with rank = the reference's depth-first leaf order.
#pragma once

#include "spt_internal.h"
#include "traverse.cuh"

namespace spt {

constexpr int kWideStack = 32;

__device__ __forceinline__ uint32_t byte_of(uint32_t lo, uint32_t hi, int j) {
    return ((j < 4 ? lo : hi) >> (8 * (j & 3))) & 0xFFu;
}

__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }

// A ray's 1/d has its zero components replaced by a tiny signed value, and inv_oct is its slot order
// key: slot ^ inv_oct, ascending = near to far.

__device__ __forceinline__ float safe_inv(float d) {
    return 1.0f / (fabsf(d) > 1e-20f ? d : copysignf(1e-20f, d));
}

// Minimum and maximum of three in one instruction.
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Two floats in a 64-bit register, and both products and sums in one instruction (f32x2).
__device__ __forceinline__ unsigned long long pack_f2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f2(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The byte q of child j as a float: q itself (CONVERT), or 32768 + q, the byte moved into the mantissa of
// 2^15.  A conversion takes a slot of the quarter-rate unit, a permute one of the integer unit, and the
// integer unit is the busiest pipe of the traversal (57 % of its cycles, against 21 % of the other).
template <bool CONVERT>
__device__ __forceinline__ float plane_of(uint32_t lo, uint32_t hi, int j) {
    if (CONVERT) return static_cast<float>(byte_of(lo, hi, j));
    return __uint_as_float(__byte_perm(j < 4 ? lo : hi, 0x47000000u, 0x7404u | ((j & 3) << 4)));
}

// A mask of slots with bit j moved to bit j ^ inv_oct: ascending bits are near to far.
__device__ __forceinline__ uint32_t near_first(uint32_t m, uint32_t inv_oct) {
    if (inv_oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
    if (inv_oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
    if (inv_oct & 4u) m = ((m & 0x0Fu) << 4) | (m >> 4);
    return m;
}

// A child is met if its far planes lie behind its near ones by more than rounding can have turned round: the
// nearest far plane, times 1 + kBoxSlack, not before the farthest near one (after Ize, "Robust BVH Ray
// Traversal", JCGT 2013).  A hit at t lies between the exact planes, so the computed ones have tmin <=
// t (1 + 5 x 2^-24) and tmax >= t (1 - 5 x 2^-24), and the hit point that the reference's inside test
// takes is rounded by 2 x 2^-24 of t on either side: 14 x 2^-24 in all, of which kBoxSlack is more than
// twice.  (Also of the offset's 255 steps at most, which a converted plane has no margin for: 3 x 2^-24
// of the node's extent, against the 1e-3 by which the reference's boxes are inflated.)  Without it, rays
// from far away lost hits: of 2^22 against 1.31M triangles, 2 from 3,000 units, 12 from 6,000, 32 from 8,000;
// with it none, from 20,000 units either (where the reference's own box test loses hundreds of them).
// The product takes the place of a subtraction, so it costs no instruction: 2^24 incoherent rays 2.98 ms
// either way.
constexpr float kBoxSlack = 1.0f / 524288.0f;   // 2^-19
__device__ __forceinline__ float boxes_meet(float tmin, float tmax) {   // the sign: not met
    return __fmaf_rn(tmax, 1.0f + kBoxSlack, -tmin);
}

// The children of node idx that the ray (o, 1/d) meets before best_t: inner children as near-to-far
// bits in `hits` (with the node's inner mask and first child), triangles as bits of t_mask from t_base.
//
// A child's plane lies at t = (p - o) / d + q 2^e / d, one fused multiply-add.  With 32768 + q in q's
// place the offset (p - o) / d moves by 32768 steps.  Its rounding is then at most 2^-24 of the offset and
// 2^-9 of a step: the near planes are moved 2^-8 of a step towards the ray's origin and the far planes
// away from it (both factors, 32768 +- 2^-8, are exact), and what grows with the distance, here and in
// the offset, 1/d and the multiply-add, at most 5 x 2^-24 of t, is kBoxSlack's (boxes_meet).
// The box test bounds a visit by its instructions: converting, scaling and comparing 48 planes.  Near
// and far plane of a child and axis go through one packed multiply-add; the hits gather as sign bits
// (boxes_meet) in a mask by slot, which is split into inner children and leaves once; x is converted
// and y and z are permuted where the whole warp is in the node step (CONVERT_X: 2^24 incoherent rays 3.01 ms a
// call, 3.07 with x permuted too, the normal caster at 1920x1080 557 and 574 us, the layered path tracing 13.7
// and 13.8 ms).  When this test came in, a conversion and a multiply-add per plane and both masks built per
// child took 4 % more on the 2^24 rays, 10 % on 300,007.
template <bool CONVERT_X>
__device__ __forceinline__ void wide_node_hits(const uint4* wnode, V3 o, float ix, float iy, float iz,
                                               uint32_t inv_oct, uint32_t idx, float best_t, uint32_t& g_base,
                                               uint32_t& g_hits, uint32_t& g_imask, uint32_t& t_base,
                                               uint32_t& t_mask) {
    const uint4* n = wnode + 5ull * idx;
    const uint4 w0 = __ldg(n), w1 = __ldg(n + 1), w2 = __ldg(n + 2), w3 = __ldg(n + 3), w4 = __ldg(n + 4);
    const int ex = static_cast<int8_t>(w0.w & 0xFFu), ey = static_cast<int8_t>((w0.w >> 8) & 0xFFu),
              ez = static_cast<int8_t>((w0.w >> 16) & 0xFFu);
    const uint32_t imask = w0.w >> 24;
    const float sx = exp2i(ex) * ix, sy = exp2i(ey) * iy, sz = exp2i(ez) * iz;
    const float ox = (__uint_as_float(w0.x) - o.x) * ix;
    const float oy = (__uint_as_float(w0.y) - o.y) * iy;
    const float oz = (__uint_as_float(w0.z) - o.z) * iz;
    const float ex2 = copysignf(0.00390625f, ix), ey2 = copysignf(0.00390625f, iy), ez2 = copysignf(0.00390625f, iz);
    const unsigned long long s2x = pack_f2(sx, sx), s2y = pack_f2(sy, sy), s2z = pack_f2(sz, sz);
    const unsigned long long o2x = CONVERT_X ? pack_f2(ox, ox)
                                             : pack_f2(__fmaf_rn(sx, -32768.0f - ex2, ox), __fmaf_rn(sx, ex2 - 32768.0f, ox));
    const unsigned long long o2y = pack_f2(__fmaf_rn(sy, -32768.0f - ey2, oy), __fmaf_rn(sy, ey2 - 32768.0f, oy));
    const unsigned long long o2z = pack_f2(__fmaf_rn(sz, -32768.0f - ez2, oz), __fmaf_rn(sz, ez2 - 32768.0f, oz));
    // The near plane is the low plane when 1/d >= 0.  The choice is made once per node on whole
    // words (four children's planes each), not per child and plane: 12 selects instead of 48.
    const bool nx = ix >= 0.0f, ny = iy >= 0.0f, nz = iz >= 0.0f;
    const uint32_t nx0 = nx ? w2.x : w3.z, nx1 = nx ? w2.y : w3.w, fx0 = nx ? w3.z : w2.x, fx1 = nx ? w3.w : w2.y;
    const uint32_t ny0 = ny ? w2.z : w4.x, ny1 = ny ? w2.w : w4.y, fy0 = ny ? w4.x : w2.z, fy1 = ny ? w4.y : w2.w;
    const uint32_t nz0 = nz ? w3.x : w4.z, nz1 = nz ? w3.y : w4.w, fz0 = nz ? w4.z : w3.x, fz1 = nz ? w4.w : w3.y;
    uint32_t missed = 0;
#pragma unroll
    for (int j = 7; j >= 0; --j) {
        float tnx, tfx, tny, tfy, tnz, tfz;
        unpack_f2(fma_f2(pack_f2(plane_of<CONVERT_X>(nx0, nx1, j), plane_of<CONVERT_X>(fx0, fx1, j)), s2x, o2x), tnx, tfx);
        unpack_f2(fma_f2(pack_f2(plane_of<false>(ny0, ny1, j), plane_of<false>(fy0, fy1, j)), s2y, o2y), tny, tfy);
        unpack_f2(fma_f2(pack_f2(plane_of<false>(nz0, nz1, j), plane_of<false>(fz0, fz1, j)), s2z, o2z), tnz, tfz);
        const float tmin = fmaxf(max3(tnx, tny, tnz), 0.0f);
        const float tmax = fminf(min3(tfx, tfy, tfz), best_t);
        missed = __funnelshift_l(__float_as_uint(boxes_meet(tmin, tmax)), missed, 1);   // its sign
    }
    const uint32_t met = ~missed & 0xFFu;
    const uint32_t hits = near_first(met & imask, inv_oct);
    // leaves (an empty slot has meta 0, which adds no triangle)
    uint32_t tm = 0;
    for (uint32_t l = met & ~imask; l; l &= l - 1) {
        const uint32_t meta = __byte_perm(w1.z, w1.w, __ffs(l) - 1) & 0xFFu;
        tm |= (meta >> 5) << (meta & 31u);
    }
    g_base = w1.x;
    g_hits = hits;
    g_imask = imask;
    t_base = w1.y;
    t_mask = tm;
}

// One candidate triangle/sphere.  Without `exact`, the reference's inside-the-leaf-box test is
// deferred to the final hit (persistent_trace / closest_hit_wide): a candidate that beats the
// current best on (t, rank) is kept either way, and if the final hit fails the test the ray is traced
// again with the test applied to every candidate.  Pruning with a best t that might later be rejected
// is safe because the final best, once it passes, is the minimum over all candidates with t > 0.
__device__ __forceinline__ void wide_candidate(const DevScene& S, uint32_t wslot, V3 o, V3 d, Hit1& h, bool exact) {
    const float4 a = __ldg(S.wtri + 3 * wslot);
    const float4 b = __ldg(S.wtri + 3 * wslot + 1);
    const float4 c = __ldg(S.wtri + 3 * wslot + 2);
    const uint32_t rank = __float_as_uint(a.w);
    float t, u = 0.0f, v = 0.0f;
    const bool sphere = (__float_as_uint(c.w) >> 31) != 0u;
    const bool ok = sphere ? sphere_test(f3v(a), c.x, o, d, t) : tri_test(f3v(a), f3v(b), f3v(c), o, d, t, u, v);
    if (!ok || !(t > 0.0f)) return;
    if (!(t < h.t || (h.found && t == h.t && rank < h.slot))) return;
    const uint32_t leaf = __float_as_uint(c.w) & 0x7FFFFFFFu;
    if (exact && !inside(S.leaf_box + 6 * leaf, hit_pos(sphere, o, d, t))) return;
    h.t = t;
    h.u = u;
    h.v = v;
    h.slot = rank;
    h.leaf = leaf;
    h.found = true;
}

// The deferred inside test of the final hit (o + d*t is the same float expression for both
// primitive kinds).
__device__ __forceinline__ bool final_inside(const DevScene& S, const Hit1& h, V3 o, V3 d) {
    return !h.found || inside(S.leaf_box + 6 * h.leaf, o + d * h.t);
}

__device__ __forceinline__ Hit1 closest_hit_wide_pass(const DevScene& S, V3 o, V3 d, uint32_t* overflow, bool exact) {
    Hit1 h;
    h.t = inf_f();
    h.u = h.v = 0.0f;
    h.slot = 0;
    h.leaf = 0;
    h.found = false;
    if (S.empty) return h;
    if (S.no_accel) {
        for (uint32_t s = 0; s < S.n_prims; ++s) prim_candidate(S, s, nullptr, o, d, false, h);
        return h;
    }
    {
        const RayInv ri = ray_inv(o, d);
        float t0, t1;
        if (!slab(ri, S.root_min[0], S.root_min[1], S.root_min[2], S.root_max[0], S.root_max[1], S.root_max[2], t0,
                  t1))
            return h;
    }
    const float ix = safe_inv(d.x), iy = safe_inv(d.y), iz = safe_inv(d.z);
    const uint32_t inv_oct = (ix >= 0.0f ? 0u : 1u) | (iy >= 0.0f ? 0u : 2u) | (iz >= 0.0f ? 0u : 4u);
    uint2 stack[kWideStack];
    int sp = 0;
    uint32_t g_base, g_hits, g_imask, t_base, t_mask;
    wide_node_hits<false>(S.wnode, o, ix, iy, iz, inv_oct, 0, h.t, g_base, g_hits, g_imask, t_base, t_mask);
    for (;;) {
        while (t_mask) {
            const int k = __ffs(t_mask) - 1;
            t_mask &= t_mask - 1;
            wide_candidate(S, t_base + k, o, d, h, exact);
        }
        if (!g_hits) {
            if (sp == 0) break;
            const uint2 e = stack[--sp];   // one 8-byte load
            g_base = e.x;
            g_hits = e.y & 0xFFu;
            g_imask = e.y >> 8;
        }
        const uint32_t key = __ffs(g_hits) - 1;
        g_hits &= g_hits - 1;
        const uint32_t s = key ^ inv_oct;
        const uint32_t child = g_base + __popc(g_imask & ((1u << s) - 1u));
        if (g_hits) {
            if (sp < kWideStack) {
                stack[sp] = make_uint2(g_base, g_hits | (g_imask << 8));
                ++sp;
            } else {
                atomicOr(overflow, 1u);
            }
        }
        wide_node_hits<false>(S.wnode, o, ix, iy, iz, inv_oct, child, h.t, g_base, g_hits, g_imask, t_base, t_mask);
    }
    return h;
}

__device__ __forceinline__ Hit1 closest_hit_wide(const DevScene& S, V3 o, V3 d, uint32_t* overflow) {
    Hit1 h = closest_hit_wide_pass(S, o, d, overflow, false);
    if (!final_inside(S, h, o, d)) h = closest_hit_wide_pass(S, o, d, overflow, true);
    return h;
}

// ---- the same traversal by a warp for 32 rays at a time ----------------------------------------
//
// Each lane walks its own ray's nodes; the triangles the lanes come across go to a queue in shared
// memory, and whenever 32 have gathered the whole warp tests them, one triangle per lane, whichever
// lanes' rays they belong to.  What bounds the traversal is the number of instructions a warp issues
// for its lanes (the nodes and triangles sit in L1 and L2): a triangle test by the lane that met it
// runs with the few lanes that met one in the same step, a queued one with all 32.
//
// Two consequences.  A ray keeps walking while its triangles wait, pruned by a best t that does not
// know them yet: more node visits, never a different answer, since the answer is the minimum of
// (t, rank) over every candidate and a stale best t is only ever too large.  And a ray is finished
// when it has no node left and its last queued triangle has been tested.
//
// On 2^24 incoherent rays against 1.31M triangles the call (order and gather included) takes 2.99 ms, and
// took 5.14 with each lane testing its own triangles and the lane's state in local memory; 300,007 rays
// 161 against 372 us.
//
// The per-lane node stack is an array of its own, not a member of the lane's state: a dynamically
// indexed member keeps the whole struct around it in local memory (the kernels that had it so read
// and wrote about eleven local words per node visit, more than their node and triangle loads).
//
// The lane's best hit sits in shared memory, where the lane that tested the triangle writes it: the
// 64-bit key t << 32 | rank (t > 0, so its bits order as t does) takes the minimum atomically, and the
// lane whose key stands writes the barycentrics, the primitive and the leaf.
constexpr uint32_t kQueue = 128;   // entries, a power of two of at least 64
struct WarpQueue {
    unsigned long long entry[kQueue];   // triangle record's address | owner lane << 59
    unsigned long long key[32];
    float2 uv[32];
    uint2 id[32];                       // primitive, leaf
    uint32_t tail;                      // one past the newest entry (the same as the warp's qtail)
    uint32_t pool, pool_end;            // the warp's rays in hand
    uint32_t chunk, first;              // rays per chunk, and the first ray the counter hands out
};
// A warp stops waiting for 32 triangles once this many lanes have nothing else to do (queries and paths
// measure alike at 4, 8 and 16).
constexpr int kWait = 8;
constexpr unsigned long long kNoHitKey = 0x7F800000FFFFFFFFull;   // t = +inf, any rank

// What the traversal reads of a scene: pointers that stay in the constant bank for a kernel of one
// scene, or in registers where every lane may have its own.
struct WideScene {
    const uint4* wnode;
    const float4* wtri;
    const float* leaf_box;
};
__device__ __forceinline__ WideScene wide_scene(const DevScene& S) { return WideScene{S.wnode, S.wtri, S.leaf_box}; }

// One lane's ray, without its node stack.  COUNT adds the lane's work (node visits, primitive tests).
template <int DEPTH, bool COUNT = false>
struct LaneTrace {
    static_assert(DEPTH >= 1 && DEPTH <= kWideStack, "stack depth out of range");
    V3 o, d;
    float ix, iy, iz;
    uint32_t inv_oct;
    float best_t;
    uint32_t g_base, g_bits;   // pending children of one node: first child, hits (near first) | inner mask << 8
    int sp;
    uint32_t last;             // one past the queue position of the ray's newest triangle
    bool has, exact;
    uint32_t n_nodes, n_prims;

    __device__ __forceinline__ void clear() {
        has = exact = false;
        g_base = g_bits = 0;
        sp = 0;
        last = 0;
        best_t = inf_f();
        o = d = v3(0.0f, 0.0f, 0.0f);
        ix = iy = iz = 0.0f;
        inv_oct = 0;
        n_nodes = n_prims = 0;
    }
    __device__ __forceinline__ bool walking() const { return (g_bits & 0xFFu) != 0u || sp > 0; }

    // From the first node again, with the lane's o and d (in exact mode after a failed inside test).
    __device__ __forceinline__ void restart(WarpQueue& Q, uint32_t qhead, bool exact_) {
        exact = exact_;
        best_t = inf_f();
        sp = 0;
        last = qhead;
        g_base = 0;                          // a pending visit of node 0: one hit child (slot 0, whose
        g_bits = (1u << inv_oct) | (1u << 8);   // near-to-far key is inv_oct) of a parent of node 0
        Q.key[threadIdx.x & 31u] = kNoHitKey;
    }

    // Takes a ray; false when the scene's root box (the reference's own slab test) is missed.  The root
    // node is visited by the next step, together with the other lanes' node visits.
    __device__ __forceinline__ bool start(const float* root_min, const float* root_max, V3 o_, V3 d_, WarpQueue& Q,
                                          uint32_t qhead) {
        o = o_;
        d = d_;
        const RayInv ri = ray_inv(o, d);
        float t0, t1;
        has = slab(ri, root_min[0], root_min[1], root_min[2], root_max[0], root_max[1], root_max[2], t0, t1);
        if (!has) return false;
        // safe_inv without dividing again: 1/d is already in ri unless |d| <= 1e-20
        ix = fabsf(d.x) > 1e-20f ? ri.inv.x : copysignf(1.0f / 1e-20f, d.x);
        iy = fabsf(d.y) > 1e-20f ? ri.inv.y : copysignf(1.0f / 1e-20f, d.y);
        iz = fabsf(d.z) > 1e-20f ? ri.inv.z : copysignf(1.0f / 1e-20f, d.z);
        inv_oct = (ix >= 0.0f ? 0u : 1u) | (iy >= 0.0f ? 0u : 2u) | (iz >= 0.0f ? 0u : 4u);
        restart(Q, qhead, false);
        return true;
    }

    // The lane's next node; its triangles come back as a run (t_base, t_mask).  A traversal that needs
    // more than `limit` stack entries sets the overflow status bit instead of pushing.
    __device__ __forceinline__ void visit(const uint4* wnode, uint2 (&stack)[DEPTH], int limit, uint32_t* status,
                                          uint32_t& t_base, uint32_t& t_mask) {
        if (!(g_bits & 0xFFu)) {
            const uint2 e = stack[--sp];   // one 8-byte load
            g_base = e.x;
            g_bits = e.y;
        }
        const uint32_t s = static_cast<uint32_t>(__ffs(g_bits) - 1) ^ inv_oct;
        g_bits &= g_bits - 1;
        const uint32_t child = g_base + __popc((g_bits >> 8) & ((1u << s) - 1u));
        if (g_bits & 0xFFu) {
            if (sp < limit) stack[sp++] = make_uint2(g_base, g_bits);
            else atomicOr(status, 1u);
        }
        uint32_t hits, imask;
        wide_node_hits<true>(wnode, o, ix, iy, iz, inv_oct, child, best_t, g_base, hits, imask, t_base, t_mask);
        g_bits = hits | (imask << 8);
        if (COUNT) ++n_nodes;
    }
};

// Tests the oldest nq <= 32 triangles of the queue, one per lane, by the whole warp.
template <int DEPTH, bool COUNT>
__device__ __forceinline__ void test_queued(WarpQueue& Q, uint32_t& qhead, uint32_t nq, const WideScene& W,
                                            LaneTrace<DEPTH, COUNT>& tr, unsigned exact_lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();   // the entries are written
    const bool mine = lane < nq;
    const unsigned long long e = Q.entry[(qhead + lane) & (kQueue - 1)];
    const uint32_t owner = mine ? static_cast<uint32_t>(e >> 59) : lane;
    const V3 o = v3(__shfl_sync(0xFFFFFFFFu, tr.o.x, owner), __shfl_sync(0xFFFFFFFFu, tr.o.y, owner),
                    __shfl_sync(0xFFFFFFFFu, tr.o.z, owner));
    const V3 d = v3(__shfl_sync(0xFFFFFFFFu, tr.d.x, owner), __shfl_sync(0xFFFFFFFFu, tr.d.y, owner),
                    __shfl_sync(0xFFFFFFFFu, tr.d.z, owner));
    const float* box = W.leaf_box;
    if (exact_lanes)   // rare: the owner's scene for the inside test
        box = reinterpret_cast<const float*>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(box), owner));
    qhead += nq;
    bool ok = false;
    float t = 0.0f, u = 0.0f, v = 0.0f;
    uint32_t prim = 0, leaf = 0;
    unsigned long long key = 0;
    if (mine) {
        const float4* p = reinterpret_cast<const float4*>(e & ((1ull << 59) - 1));
        const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
        prim = __float_as_uint(b.w);
        leaf = __float_as_uint(c.w) & 0x7FFFFFFFu;
        const bool sphere = (__float_as_uint(c.w) >> 31) != 0u;
        ok = sphere ? sphere_test(f3v(a), c.x, o, d, t) : tri_test(f3v(a), f3v(b), f3v(c), o, d, t, u, v);
        key = (static_cast<unsigned long long>(__float_as_uint(t)) << 32) | __float_as_uint(a.w);
        ok = ok && t > 0.0f && t < inf_f() && key < Q.key[owner];
        if (ok && ((exact_lanes >> owner) & 1u)) ok = inside(box + 6ull * leaf, hit_pos(sphere, o, d, t));
        if (COUNT) ++tr.n_prims;
    }
    __syncwarp();   // entries and keys are read
    if (__any_sync(0xFFFFFFFFu, ok)) {
        if (ok) atomicMin(&Q.key[owner], key);
        __syncwarp();
        if (ok && Q.key[owner] == key) {   // ranks are unique, so one lane per owner
            Q.uv[owner] = make_float2(u, v);
            Q.id[owner] = make_uint2(prim, leaf);
        }
        __syncwarp();
        tr.best_t = __uint_as_float(static_cast<uint32_t>(Q.key[lane] >> 32));
    }
}

// One step of the warp: every walking lane visits a node, and the triangles found are queued and
// tested 32 at a time.
template <int DEPTH, bool COUNT>
__device__ __forceinline__ void warp_step(WarpQueue& Q, uint32_t& qhead, uint32_t& qtail, const WideScene& W,
                                          LaneTrace<DEPTH, COUNT>& tr, uint2 (&stack)[DEPTH], int limit,
                                          uint32_t* status, unsigned exact_lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t t_base = 0, t_mask = 0;
    if (tr.walking()) tr.visit(W.wnode, stack, limit, status, t_base, t_mask);
    // Room for all of them (31 at most are left over, and a step finds 15 on average): each lane reserves a
    // run of places with one shared-memory atomic and fills it.  Otherwise one triangle per lane at a
    // time, with tests in between.  (Appending one per lane at a time throughout takes six rounds of
    // ballots a step: 3.38 against 3.01 ms a call on 2^24 incoherent rays, the layered path tracing 14.8
    // against 13.7 ms, the normal caster 648 against 557 us.)
    const uint32_t mine = __popc(t_mask), all = __reduce_add_sync(0xFFFFFFFFu, mine);
    if (!all) return;
    const unsigned long long first =
        reinterpret_cast<unsigned long long>(W.wtri + 3ull * t_base) | (static_cast<unsigned long long>(lane) << 59);
    if (qtail - qhead + all <= kQueue) {
        if (mine) {
            uint32_t pos = atomicAdd(&Q.tail, mine);
            tr.last = pos + mine;
            for (; t_mask; t_mask &= t_mask - 1, ++pos)
                Q.entry[pos & (kQueue - 1)] = first + static_cast<uint32_t>(__ffs(t_mask) - 1) * (3u * sizeof(float4));
        }
        qtail += all;
    }
    for (;;) {
        while (qtail - qhead >= 32) test_queued(Q, qhead, 32u, W, tr, exact_lanes);
        const unsigned found = __ballot_sync(0xFFFFFFFFu, t_mask != 0u);
        if (!found) return;
        if (t_mask) {
            const uint32_t pos = qtail + __popc(found & ((1u << lane) - 1u));
            Q.entry[pos & (kQueue - 1)] = first + static_cast<uint32_t>(__ffs(t_mask) - 1) * (3u * sizeof(float4));
            t_mask &= t_mask - 1;
            tr.last = pos + 1;
        }
        qtail += __popc(found);
        __syncwarp();   // earlier steps' reservations (votes and reductions order no memory)
        if (lane == 0) Q.tail = qtail;
        __syncwarp();
    }
}

// The queue's rest tested, if enough of the lanes that do not walk wait for it (or none walks).
template <int DEPTH, bool COUNT>
__device__ __forceinline__ void test_rest(WarpQueue& Q, uint32_t& qhead, uint32_t qtail, const WideScene& W,
                                          LaneTrace<DEPTH, COUNT>& tr, unsigned walkers, unsigned exact_lanes) {
    if (qtail == qhead) return;
    const unsigned waits = __ballot_sync(0xFFFFFFFFu, tr.has && !tr.walking() && static_cast<int>(qhead - tr.last) < 0);
    if (__popc(waits) >= kWait || !walkers) test_queued(Q, qhead, qtail - qhead, W, tr, exact_lanes);
}

// Persistent warps with dynamic ray fetch (after Aila & Laine, "Understanding the Efficiency of Ray
// Traversal on GPUs", HPG 2009): a lane whose ray is finished takes the next ray at once instead of
// idling until the warp's longest ray ends.  Ray indices come from a warp-local pool refilled `chunk`
// at a time from one global counter, so the counter sees one atomic per chunk.  2^24 rays take 3.08 / 3.01 / 3.00
// / 3.06 ms at 16 / 32 / 64 / 128 rays per chunk, the layered path tracing 13.6 / 13.7 / 14.5 / 15.9, the box 1.29
// / 1.30 / 1.34 / 1.45 (a shorter tail, and the ordered neighbours stay together).
constexpr uint32_t kChunk = 32;
// Lanes are served (hit stored, next ray taken) once this many wait, or no lane is busy: the branch runs
// with the waiting lanes only.  2^24 rays take 3.30 / 3.14 / 3.01 / 3.01 / 3.10 ms at 2 / 4 / 8 / 12 / 16.
constexpr int kRefill = 8;

// source: load(i, o, d) fetches ray i (and, for a kernel of many scenes, the lane's scene), move(from)
// takes lane `from`'s scene, root_min() and root_max() are its scene's root box, scene() its WideScene,
// store(i, t, prim, u, v) takes the hit.

// The result of the lane's ray, all of whose candidates have been tested: stored, or false when the final
// hit fails the deferred inside test (o + d*t is the same float expression for both primitive kinds):
// the ray is then traced again, with the test applied to every candidate.
template <int DEPTH, bool COUNT, typename Source>
__device__ __forceinline__ bool settle(const WarpQueue& Q, Source& src, const LaneTrace<DEPTH, COUNT>& tr, uint32_t ray) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long key = Q.key[lane];
    if (key == kNoHitKey) {
        src.store(ray, inf_f(), SPT_MISS, 0.0f, 0.0f);
        return true;
    }
    const float t = __uint_as_float(static_cast<uint32_t>(key >> 32));
    const uint2 id = Q.id[lane];
    if (!tr.exact && !inside(src.scene().leaf_box + 6ull * id.y, tr.o + tr.d * t)) return false;
    const float2 uv = Q.uv[lane];
    src.store(ray, t, id.x, uv.x, uv.y);
    return true;
}

// The warp's last rays, four at most: eight lanes to a ray, one child of its node each.  A lone lane's
// visit is a chain of some 400 instructions, most of them the eight children's box tests one after the
// other; a batch of a few rays per warp, and the end of any batch, waits for such chains (the longest
// ray of 1,000 incoherent ones visits 88 nodes: alone it took 80 us, here 55).  300,007 rays against 1.31M
// triangles take 161 us instead of 203, the layered path tracing 13.7 ms instead of 14.6, the normal caster 557
// us instead of 581.  The lanes of a group hold copies of the ray's state; the first of them, its leader,
// keeps the node stack, the best hit and the queue entries' name.
constexpr int kLast = 4;
template <int DEPTH, bool COUNT, typename Source>
__device__ __forceinline__ void trace_last(WarpQueue& Q, Source& src, LaneTrace<DEPTH, COUNT>& tr, uint2 (&stack)[DEPTH],
                                           uint32_t ray, uint32_t qhead, uint32_t qtail, int limit, uint32_t* status,
                                           unsigned exact_lanes) {
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u, leader = lane & ~7u;
    // the queue first: its entries name the lanes as they are now
    while (qtail != qhead) test_queued(Q, qhead, min(qtail - qhead, 32u), src.scene(), tr, exact_lanes);
    {
        unsigned m = __ballot_sync(kAll, tr.has);
        for (uint32_t g = 0; g < (lane >> 3); ++g) m &= m - 1;
        const bool live = m != 0u;
        const uint32_t from = live ? __ffs(m) - 1 : lane;
        tr.exact = live && ((exact_lanes >> from) & 1u);
        tr.o = v3(__shfl_sync(kAll, tr.o.x, from), __shfl_sync(kAll, tr.o.y, from), __shfl_sync(kAll, tr.o.z, from));
        tr.d = v3(__shfl_sync(kAll, tr.d.x, from), __shfl_sync(kAll, tr.d.y, from), __shfl_sync(kAll, tr.d.z, from));
        tr.ix = __shfl_sync(kAll, tr.ix, from);
        tr.iy = __shfl_sync(kAll, tr.iy, from);
        tr.iz = __shfl_sync(kAll, tr.iz, from);
        tr.inv_oct = __shfl_sync(kAll, tr.inv_oct, from);
        tr.g_base = __shfl_sync(kAll, tr.g_base, from);
        tr.g_bits = __shfl_sync(kAll, tr.g_bits, from);
        tr.sp = __shfl_sync(kAll, tr.sp, from);
        ray = __shfl_sync(kAll, ray, from);
        src.move(from);
        tr.has = live;
        if (!live) {
            tr.g_bits = 0;
            tr.sp = 0;
        }
        const int deepest = __reduce_max_sync(kAll, tr.sp);
        for (int i = 0; i < deepest; ++i) {   // every lane reads entry i before any leader writes it
            const uint2 e = stack[i];
            const uint32_t x = __shfl_sync(kAll, e.x, from), y = __shfl_sync(kAll, e.y, from);
            if (sub == 0) stack[i] = make_uint2(x, y);
        }
        const unsigned long long key = Q.key[from];
        const float2 uv = Q.uv[from];
        const uint2 id = Q.id[from];
        __syncwarp();
        if (sub == 0) {
            Q.key[lane] = key;
            Q.uv[lane] = uv;
            Q.id[lane] = id;
        }
        __syncwarp();
        tr.best_t = __uint_as_float(static_cast<uint32_t>(key >> 32));
    }
    for (;;) {
        exact_lanes = __ballot_sync(kAll, sub == 0 && tr.exact);
        for (;;) {
            const bool walks = tr.walking();   // the same in all lanes of a group
            if (!__any_sync(kAll, walks)) break;
            const bool pop = walks && !(tr.g_bits & 0xFFu);
            if (__any_sync(kAll, pop)) {
                uint2 e = make_uint2(0u, 0u);
                if (pop && sub == 0) e = stack[tr.sp - 1];
                e.x = __shfl_sync(kAll, e.x, leader);
                e.y = __shfl_sync(kAll, e.y, leader);
                if (pop) {
                    tr.g_base = e.x;
                    tr.g_bits = e.y;
                    --tr.sp;
                }
            }
            const WideScene W = src.scene();
            bool hit = false;
            uint32_t meta = 0, imask = 0, t_base = 0;
            if (walks) {
                const uint32_t s = static_cast<uint32_t>(__ffs(tr.g_bits) - 1) ^ tr.inv_oct;
                tr.g_bits &= tr.g_bits - 1;
                const uint32_t child = tr.g_base + __popc((tr.g_bits >> 8) & ((1u << s) - 1u));
                if (tr.g_bits & 0xFFu) {
                    if (tr.sp < limit) {
                        if (sub == 0) stack[tr.sp] = make_uint2(tr.g_base, tr.g_bits);
                        ++tr.sp;
                    } else if (sub == 0) {
                        atomicOr(status, 1u);
                    }
                }
                // this lane's child: the box test of wide_node_hits
                const uint4* nd = W.wnode + 5ull * child;
                const uint8_t* q = reinterpret_cast<const uint8_t*>(nd + 2) + sub;
                const bool px = tr.ix >= 0.0f, py = tr.iy >= 0.0f, pz = tr.iz >= 0.0f;
                const float nx = __ldg(q + (px ? 0 : 24)), fx = __ldg(q + (px ? 24 : 0));
                const float ny = __ldg(q + (py ? 8 : 32)), fy = __ldg(q + (py ? 32 : 8));
                const float nz = __ldg(q + (pz ? 16 : 40)), fz = __ldg(q + (pz ? 40 : 16));
                const uint4 w0 = __ldg(nd), w1 = __ldg(nd + 1);
                const float sx = exp2i(static_cast<int8_t>(w0.w & 0xFFu)) * tr.ix;
                const float sy = exp2i(static_cast<int8_t>((w0.w >> 8) & 0xFFu)) * tr.iy;
                const float sz = exp2i(static_cast<int8_t>((w0.w >> 16) & 0xFFu)) * tr.iz;
                const float ox = (__uint_as_float(w0.x) - tr.o.x) * tr.ix;
                const float oy = (__uint_as_float(w0.y) - tr.o.y) * tr.iy;
                const float oz = (__uint_as_float(w0.z) - tr.o.z) * tr.iz;
                const float tmin = fmaxf(max3(__fmaf_rn(nx, sx, ox), __fmaf_rn(ny, sy, oy), __fmaf_rn(nz, sz, oz)), 0.0f);
                const float tmax = fminf(min3(__fmaf_rn(fx, sx, ox), __fmaf_rn(fy, sy, oy), __fmaf_rn(fz, sz, oz)), tr.best_t);
                hit = !(__float_as_uint(boxes_meet(tmin, tmax)) >> 31);
                meta = byte_of(sub < 4 ? w1.z : w1.w, 0u, sub & 3u);
                imask = w0.w >> 24;
                tr.g_base = w1.x;
                t_base = w1.y;
            }
            const uint32_t met = (__ballot_sync(kAll, hit) >> leader) & 0xFFu;
            if (walks) tr.g_bits = near_first(met & imask, tr.inv_oct) | (imask << 8);
            const bool leaf = hit && !((imask >> sub) & 1u);
            const uint32_t cnt = leaf ? __popc(meta >> 5) : 0u, all = __reduce_add_sync(kAll, cnt);
            if (all) {   // at most 4 x 24, behind at most 31: the queue holds them
                if (cnt) {
                    const uint32_t pos = atomicAdd(&Q.tail, cnt);
                    const unsigned long long first =
                        reinterpret_cast<unsigned long long>(W.wtri + 3ull * (t_base + (meta & 31u))) |
                        (static_cast<unsigned long long>(leader) << 59);
                    for (uint32_t k = 0; k < cnt; ++k) Q.entry[(pos + k) & (kQueue - 1)] = first + k * (3u * sizeof(float4));
                }
                qtail += all;
                while (qtail - qhead >= 32) test_queued(Q, qhead, 32u, W, tr, exact_lanes);
                tr.best_t = __uint_as_float(static_cast<uint32_t>(Q.key[leader] >> 32));
            }
            if (COUNT && walks && sub == 0) ++tr.n_nodes;
        }
        if (qtail != qhead) test_queued(Q, qhead, qtail - qhead, src.scene(), tr, exact_lanes);
        bool again = false;
        if (tr.has && sub == 0) again = !settle(Q, src, tr, ray);
        tr.has = __shfl_sync(kAll, again ? 1 : 0, leader) != 0;
        if (!__any_sync(kAll, tr.has)) return;
        if (tr.has) tr.restart(Q, qhead, true);
        __syncwarp();
    }
}

template <int DEPTH, bool COUNT, typename Source>
__device__ __forceinline__ void persistent_trace(WarpQueue& Q, Source& src, uint32_t n, unsigned long long* next,
                                                 int limit, uint32_t* status, unsigned long long* counts = nullptr) {
    const uint32_t lane = threadIdx.x & 31u;
    uint2 stack[DEPTH];
    LaneTrace<DEPTH, COUNT> tr;
    tr.clear();
    uint32_t qhead = 0, qtail = 0, mine = 0;
    if (lane == 0) {
        Q.tail = 0;
        // Small batches spread over the warps, so that a ray's chain of dependent loads has a warp for
        // itself.  A warp's first chunk goes by its number; the counter hands out those after.
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        const uint32_t chunk = min(kChunk, max(1u, n / warps));
        Q.chunk = chunk;
        Q.first = warps * chunk;
        Q.pool = min(n, (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * chunk);
        Q.pool_end = min(n, Q.pool + chunk);
    }
    __syncwarp();
    unsigned exact_lanes = 0;
    bool exhausted = false;
    for (;;) {
        const bool fin = tr.has && !tr.walking() && static_cast<int>(qhead - tr.last) >= 0;
        const unsigned need = __ballot_sync(0xFFFFFFFFu, fin || (!tr.has && !exhausted));
        const unsigned busy = __ballot_sync(0xFFFFFFFFu, tr.has && !fin);
        if (need && (__popc(need) >= kRefill || __popc(busy) <= kLast)) {
            if (fin) {
                if (settle(Q, src, tr, mine)) tr.has = false;
                else tr.restart(Q, qhead, true);
            }
            const bool want = !tr.has && !exhausted;
            const unsigned wants = __ballot_sync(0xFFFFFFFFu, want);
            const uint32_t pool = Q.pool, have = Q.pool_end - pool;
            const uint32_t cnt = __popc(wants), rank = __popc(wants & ((1u << lane) - 1u));
            uint32_t fresh = 0, extra = 0;
            bool dry = true;   // the counter has no more
            if (have < cnt && Q.first < n) {
                const uint32_t chunk = Q.chunk;
                unsigned long long f = 0;
                if (lane == 0) f = atomicAdd(next, static_cast<unsigned long long>(chunk));
                f = __shfl_sync(0xFFFFFFFFu, f, 0) + Q.first;
                dry = f + chunk >= n;
                if (f < n) {
                    fresh = static_cast<uint32_t>(f);
                    extra = min(chunk, n - fresh);
                }
            }
            if (want) {
                if (rank < have + extra) {
                    mine = rank < have ? pool + rank : fresh + (rank - have);
                    V3 o, d;
                    src.load(mine, o, d);
                    if (!tr.start(src.root_min(), src.root_max(), o, d, Q, qhead))
                        src.store(mine, inf_f(), SPT_MISS, 0.0f, 0.0f);
                } else {
                    exhausted = dry;
                }
            }
            __syncwarp();
            if (lane == 0) {
                Q.pool = have < cnt ? fresh + min(cnt - have, extra) : pool + cnt;
                if (have < cnt) Q.pool_end = fresh + extra;
            }
            __syncwarp();
            exact_lanes = __ballot_sync(0xFFFFFFFFu, tr.has && tr.exact);
            if (__all_sync(0xFFFFFFFFu, tr.has || exhausted) && __popc(__ballot_sync(0xFFFFFFFFu, tr.has)) <= kLast) break;
        }
        warp_step(Q, qhead, qtail, src.scene(), tr, stack, limit, status, exact_lanes);
        if (qtail != qhead) test_rest(Q, qhead, qtail, src.scene(), tr, __ballot_sync(0xFFFFFFFFu, tr.walking()), exact_lanes);
    }
    if (__any_sync(0xFFFFFFFFu, tr.has)) trace_last(Q, src, tr, stack, mine, qhead, qtail, limit, status, exact_lanes);
    if (COUNT) {
        unsigned long long a = tr.n_nodes, b = tr.n_prims;
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xFFFFFFFFu, a, o);
            b += __shfl_xor_sync(0xFFFFFFFFu, b, o);
        }
        if (lane == 0) {
            atomicAdd(counts, a);
            atomicAdd(counts + 1, b);
        }
    }
}

// Closest hits of one ray per lane (valid lanes only), without refill: for rays that stay together on
// their own (camera rays of a tile).
template <int DEPTH, typename Source>
__device__ __forceinline__ void trace_tile(WarpQueue& Q, Source& src, bool valid, V3 o, V3 d, uint32_t ray,
                                           uint32_t* status) {
    uint2 stack[DEPTH];
    LaneTrace<DEPTH> tr;
    tr.clear();
    uint32_t qhead = 0, qtail = 0;
    unsigned exact_lanes = 0;
    if ((threadIdx.x & 31u) == 0) Q.tail = 0;
    if (valid && !tr.start(src.root_min(), src.root_max(), o, d, Q, qhead)) src.store(ray, inf_f(), SPT_MISS, 0.0f, 0.0f);
    __syncwarp();
    unsigned rays = __ballot_sync(0xFFFFFFFFu, tr.has);
    for (;;) {
        // a step in which few lanes are out of nodes goes straight to the next visits (526 us for a 1080p
        // image, 561 with the looks below taken at every step; the refilling loop above is level or slower)
        const unsigned walkers = __ballot_sync(0xFFFFFFFFu, tr.walking());
        if (__popc(rays & ~walkers) >= kRefill || __popc(walkers) <= kLast) {
            test_rest(Q, qhead, qtail, src.scene(), tr, walkers, exact_lanes);
            const bool fin = tr.has && !tr.walking() && static_cast<int>(qhead - tr.last) >= 0;
            const unsigned ends = __ballot_sync(0xFFFFFFFFu, fin);
            if (__popc(ends) >= kRefill || __popc(rays & ~ends) <= kLast) {
                if (fin) {
                    if (settle(Q, src, tr, ray)) tr.has = false;
                    else tr.restart(Q, qhead, true);
                }
                rays = __ballot_sync(0xFFFFFFFFu, tr.has);
                exact_lanes = __ballot_sync(0xFFFFFFFFu, tr.has && tr.exact);
                if (__popc(rays) <= kLast) break;
            }
        }
        warp_step(Q, qhead, qtail, src.scene(), tr, stack, DEPTH, status, exact_lanes);
    }
    if (__any_sync(0xFFFFFFFFu, tr.has)) trace_last(Q, src, tr, stack, ray, qhead, qtail, DEPTH, status, exact_lanes);
}

// Closest hit with the traversal the scene selected (a kernel template parameter, so each kernel
// carries one traversal's registers).
template <int TRAV>
__device__ __forceinline__ Hit1 trace_closest(const DevScene& S, V3 o, V3 d, uint32_t* overflow) {
    if (TRAV >= 1) return closest_hit_wide(S, o, d, overflow);
    return closest_hit<kStack>(S, o, d, overflow);
}

}  // namespace spt
