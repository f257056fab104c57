// traverse.cuh -- ray/scene queries on the device.
//
// closest_hit(): ordered, t-pruned stack traversal of the binary SAH tree stored as 64-byte
//   "pair" nodes (both children's boxes in the parent), returning the reference's answer:
//   the reference (acceleration/sbvh.cpp:478-510) visits every node whose box passes the slab
//   test, depth first and left first, and keeps a hit iff t > 0, t < best and the hit point is
//   inside the leaf box (+-1e-3).  Its result is therefore the hit with the smallest t, ties going
//   to the leaf reference met first in depth-first order -- the smallest slot here.  The box test
//   is the reference's own (slab() in spt_device.cuh); visiting near child first and skipping
//   children with tmin > best t or tmax < 0 only drops subtrees that cannot hold a better hit:
//   every non-root box is its primitives' bounds inflated by 1e-3, so any hit inside one lies
//   at least 1e-3 / |d_axis| past the box's entry and before its exit.
//
// count_traverse(): the reference's exhaustive traversal -- no pruning -- counting box and primitive
//   tests and passes (num_intersection_tests / num_intersections, sbvh.cpp:478-510), plus the hit it
//   finds.  The counts are sums over the boxes whose parent's box passes, and the hit is the smallest
//   (t, depth-first slot) that passes the inside test, so neither depends on the order.
#pragma once

#include "spt_device.cuh"

namespace spt {

__device__ __forceinline__ float inf_f() { return __int_as_float(0x7f800000); }

struct Hit1 {
    float t, u, v;
    uint32_t slot;
    uint32_t leaf;   // reference leaf of the hit (wide traversal), for the deferred inside test
    bool found;
};

__device__ __forceinline__ void prim_candidate(const DevScene& S, uint32_t slot, const float* box, V3 o, V3 d,
                                               bool check_inside, Hit1& h) {
    const float4 a = __ldg(S.tri + 3 * slot);
    const float4 b = __ldg(S.tri + 3 * slot + 1);
    const float4 c = __ldg(S.tri + 3 * slot + 2);
    float t, u = 0.0f, v = 0.0f;
    bool sphere = __float_as_int(c.w) == SPT_PRIM_SPHERE;
    bool ok = sphere ? sphere_test(f3v(a), b.x, o, d, t) : tri_test(f3v(a), f3v(b), f3v(c), o, d, t, u, v);
    if (!ok || !(t > 0.0f)) return;
    if (!(t < h.t || (h.found && t == h.t && slot < h.slot))) return;
    if (check_inside && !inside(box, hit_pos(sphere, o, d, t))) return;
    h.t = t;
    h.u = u;
    h.v = v;
    h.slot = slot;
    h.found = true;
}

template <int STACK>
__device__ __forceinline__ Hit1 closest_hit(const DevScene& S, V3 o, V3 d, uint32_t* overflow) {
    Hit1 h;
    h.t = inf_f();
    h.u = h.v = 0.0f;
    h.slot = 0;
    h.leaf = 0;
    h.found = false;
    if (S.empty) return h;
    if (S.no_accel) {  // NoAccelStructure::intersect: every primitive, no box test, strict <
        for (uint32_t s = 0; s < S.n_prims; ++s) prim_candidate(S, s, nullptr, o, d, false, h);
        return h;
    }
    const RayInv r = ray_inv(o, d);
    float t0, t1;
    if (!slab(r, S.root_min[0], S.root_min[1], S.root_min[2], S.root_max[0], S.root_max[1], S.root_max[2], t0, t1))
        return h;
    if (S.root_is_leaf) {
        const int2 fc = __ldg(S.leaf);
        for (int k = 0; k < fc.y; ++k) prim_candidate(S, fc.x + k, S.leaf_box, o, d, true, h);
        return h;
    }
    int st_node[STACK];
    float st_t[STACK];
    int sp = 0;
    int node = 0;
    for (;;) {
        if (node >= 0) {
            const float4* p = S.pair + 4 * node;
            const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
            const int4 refs = __ldg(reinterpret_cast<const int4*>(p + 3));
            float lmin, lmax, rmin, rmax;
            bool hl = slab(r, a.x, a.y, a.z, a.w, b.x, b.y, lmin, lmax) && !(lmin > h.t) && !(lmax < 0.0f);
            bool hr = slab(r, b.z, b.w, c.x, c.y, c.z, c.w, rmin, rmax) && !(rmin > h.t) && !(rmax < 0.0f);
            if (hl && hr) {
                int near = refs.x, far = refs.y;
                float far_t = rmin;
                if (rmin < lmin) {
                    near = refs.y;
                    far = refs.x;
                    far_t = lmin;
                }
                if (sp < STACK) {
                    st_node[sp] = far;
                    st_t[sp] = far_t;
                    ++sp;
                } else {
                    atomicOr(overflow, 1u);
                }
                node = near;
                continue;
            }
            if (hl) {
                node = refs.x;
                continue;
            }
            if (hr) {
                node = refs.y;
                continue;
            }
        } else {
            const int l = ~node;
            const int2 fc = __ldg(S.leaf + l);
            for (int k = 0; k < fc.y; ++k) prim_candidate(S, fc.x + k, S.leaf_box + 6 * l, o, d, true, h);
        }
        bool got = false;
        while (sp > 0) {
            --sp;
            if (!(st_t[sp] > h.t)) {
                node = st_node[sp];
                got = true;
                break;
            }
        }
        if (!got) break;
    }
    return h;
}

struct CountOut {
    uint32_t tests, hits, prim_tests;
};

// The primitives first .. first + n - 1 of a passing leaf with box bx (NULL: no inside test).
__device__ __forceinline__ void count_leaf(const DevScene& S, uint32_t first, uint32_t n, const float* bx, V3 o, V3 d,
                                           CountOut& c, Hit1& h) {
    for (uint32_t k = 0; k < n; ++k) {
        const uint32_t s = first + k;
        const float4 a = __ldg(S.tri + 3 * s), b = __ldg(S.tri + 3 * s + 1), cc = __ldg(S.tri + 3 * s + 2);
        float t, u = 0.0f, v = 0.0f;
        bool sphere = __float_as_int(cc.w) == SPT_PRIM_SPHERE;
        bool ok = sphere ? sphere_test(f3v(a), b.x, o, d, t) : tri_test(f3v(a), f3v(b), f3v(cc), o, d, t, u, v);
        if (!ok) continue;
        ++c.hits;
        if (!(t > 0.0f) || !(t < h.t || (h.found && t == h.t && s < h.slot))) continue;
        if (bx && !inside(bx, hit_pos(sphere, o, d, t))) continue;
        h.t = t; h.u = u; h.v = v; h.slot = s; h.found = true;
    }
}

// FULL: the primitives are tested, for the passes among them and the hit; without it c.hits counts boxes
// only and no hit is returned (a test is counted whatever it finds, so the count of tests needs none).
// A step visits a pair node: both children's boxes and, for a leaf child, its primitive count, in one
// 64-byte record.  What bounds the traversal is its chain of dependent node loads and the boxes' slab
// tests; a step per box, from the tree's own 32-byte nodes, and with the primitives tested for counts
// that do not need them, took 1268 us on 1277x719 camera rays against 1.31M triangles, where this takes 350 (369
// before the rows of tiles were spread, raycast.cu).
template <int STACK, bool FULL>
__device__ __forceinline__ Hit1 count_traverse(const DevScene& S, V3 o, V3 d, CountOut& c, uint32_t* overflow) {
    Hit1 h;
    h.t = inf_f();
    h.u = h.v = 0.0f;
    h.slot = 0;
    h.leaf = 0;
    h.found = false;
    c.tests = c.hits = c.prim_tests = 0;
    if (S.empty) return h;
    if (S.no_accel) {
        c.tests = c.prim_tests = S.n_prims;
        if (FULL) count_leaf(S, 0, S.n_prims, nullptr, o, d, c, h);
        return h;
    }
    const RayInv r = ray_inv(o, d);
    float t0, t1;
    c.tests = 1;
    if (!slab(r, S.root_min[0], S.root_min[1], S.root_min[2], S.root_max[0], S.root_max[1], S.root_max[2], t0, t1))
        return h;
    c.hits = 1;
    if (S.root_is_leaf) {
        const int2 fc = __ldg(S.leaf);
        c.tests += fc.y;
        c.prim_tests = fc.y;
        if (FULL) count_leaf(S, fc.x, fc.y, S.leaf_box, o, d, c, h);
        return h;
    }
    int stack[STACK];
    int sp = 0, node = 0;
    for (;;) {
        const float4* p = S.pair + 4ull * node;
        const float4 a = __ldg(p), b = __ldg(p + 1), e = __ldg(p + 2);
        const int4 refs = __ldg(reinterpret_cast<const int4*>(p + 3));
        const bool hl = slab(r, a.x, a.y, a.z, a.w, b.x, b.y, t0, t1), hr = slab(r, b.z, b.w, e.x, e.y, e.z, e.w, t0, t1);
        c.tests += 2;
        c.hits += (hl ? 1u : 0u) + (hr ? 1u : 0u);
        if (hl && refs.x < 0) {
            c.tests += refs.z;
            c.prim_tests += refs.z;
            if (FULL) {
                const float bx[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
                count_leaf(S, __ldg(&S.leaf[~refs.x].x), refs.z, bx, o, d, c, h);
            }
        }
        if (hr && refs.y < 0) {
            c.tests += refs.w;
            c.prim_tests += refs.w;
            if (FULL) {
                const float bx[6] = {b.z, b.w, e.x, e.y, e.z, e.w};
                count_leaf(S, __ldg(&S.leaf[~refs.y].x), refs.w, bx, o, d, c, h);
            }
        }
        const bool il = hl && refs.x >= 0, ir = hr && refs.y >= 0;
        if (il || ir) {
            if (il && ir) {
                if (sp < STACK) stack[sp++] = refs.y;
                else atomicOr(overflow, 1u);
            }
            node = il ? refs.x : refs.y;
        } else {
            if (sp == 0) return h;
            node = stack[--sp];
        }
    }
}

__device__ __forceinline__ uint32_t slot_prim(const DevScene& S, uint32_t slot) {
    return __float_as_uint(__ldg(S.tri + 3 * slot).w);
}

}  // namespace spt
