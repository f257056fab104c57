// raycast.cu -- batched ray queries and the three ray-cast integrators.
//
//   k_intersect   closest hit per ray (AccelStructure::intersect, accel_structure.h:29-30)
//   k_count       the reference's exhaustive traversal: tests / passes per ray
//   k_raycast     camera ray generation fused with the query and the pixel value of one
//                 ray-caster mode (integrators/raycaster.h:62-99 + normal_raycaster.cpp:19-31,
//                 depth_raycaster.cpp:36-48, int_test_count_raycaster.cpp:75-85)
#include <algorithm>
#include <cstring>
#include <limits>

#include "spt_internal.h"
#include "traverse_wide.cuh"

namespace spt {
namespace {

constexpr int kBlock = 128;

// Ray i of a batch in either host layout: STRIDE 8 = {origin, pad, direction, pad} as two float4;
// STRIDE 6 = the reference's Ray (core/ray.h: two glm::vec3, 24 bytes) as three float2.  STREAM
// reads with the evict-first hint (rays are read once).
template <int STRIDE, bool STREAM>
__device__ __forceinline__ void load_ray(const float* __restrict__ rays, uint64_t i, V3& o, V3& d) {
    if (STRIDE == 8) {
        const float4* r = reinterpret_cast<const float4*>(rays) + 2 * i;
        const float4 a = STREAM ? __ldcs(r) : __ldg(r), b = STREAM ? __ldcs(r + 1) : __ldg(r + 1);
        o = f3v(a);
        d = f3v(b);
    } else {
        const float2* r = reinterpret_cast<const float2*>(rays) + 3 * i;
        const float2 a = STREAM ? __ldcs(r) : __ldg(r), b = STREAM ? __ldcs(r + 1) : __ldg(r + 1),
                     c = STREAM ? __ldcs(r + 2) : __ldg(r + 2);
        o = v3(a.x, a.y, b.x);
        d = v3(b.y, c.x, c.y);
    }
}

// Rays and hits of the persistent kernels.  Rays are read and hits written once, with the evict-first
// (streaming) cache hint, so the ray and hit streams (48 B per ray, 768 MB per 2^24 rays) push less of
// the scene out of L2: +1 %.  ORDERED: the k-th ray taken is order[k] (ray_order.cu) and its hit goes
// to place k, so that neighbouring lanes write neighbouring hits (scattered 16-byte stores cost
// partial-sector writes in DRAM).
template <int STRIDE, bool ORDERED>
struct RayBatch {
    const DevScene& S;
    const float* rays;
    const uint32_t* order;
    spt_hit* hits;
    __device__ __forceinline__ void load(uint32_t i, V3& o, V3& d) {
        load_ray<STRIDE, true>(rays, ORDERED ? __ldg(order + i) : i, o, d);
    }
    __device__ __forceinline__ void move(uint32_t) {}
    __device__ __forceinline__ const float* root_min() const { return S.root_min; }
    __device__ __forceinline__ const float* root_max() const { return S.root_max; }
    __device__ __forceinline__ WideScene scene() const { return wide_scene(S); }
    __device__ __forceinline__ void store(uint32_t i, float t, uint32_t prim, float u, float v) {
        __stcs(reinterpret_cast<float4*>(hits + i), make_float4(t, __uint_as_float(prim), u, v));
    }
};

// Persistent variant: wide traversal, lanes refilled from a global ray counter (traverse_wide.cuh).
// 8 blocks of 128 per SM (at most 64 registers): 2^24 incoherent rays take 3.01 ms a call at 8 blocks, 3.13 at 7, 3.37 at
// 6, 3.32 at 9 and 3.42 at 10, where the ray's state spills.
template <int STRIDE>
__global__ void __launch_bounds__(kBlock, 8) k_intersect_df(const __grid_constant__ DevScene S,
                                                         const float* __restrict__ rays, uint32_t n,
                                                         spt_hit* __restrict__ hits, uint32_t* status,
                                                         unsigned long long* next) {
    __shared__ WarpQueue q[kBlock / 32];
    RayBatch<STRIDE, false> b{S, rays, nullptr, hits};
    persistent_trace<kWideStack, false>(q[threadIdx.x >> 5], b, n, next, kWideStack, status);
}

// The same kernel over a batch in coherence order, for its first *count rays (those that meet the root
// box).
template <int STRIDE>
__global__ void __launch_bounds__(kBlock, 8) k_intersect_df_ordered(const __grid_constant__ DevScene S,
                                                                 const float* __restrict__ rays,
                                                                 const uint32_t* __restrict__ order,
                                                                 const uint32_t* __restrict__ count,
                                                                 spt_hit* __restrict__ hits_ordered, uint32_t* status,
                                                                 unsigned long long* next) {
    __shared__ WarpQueue q[kBlock / 32];
    RayBatch<STRIDE, true> b{S, rays, order, hits_ordered};
    persistent_trace<kWideStack, false>(q[threadIdx.x >> 5], b, __ldg(count), next, kWideStack, status);
}

// The same kernel with its own work counted (node visits, primitive tests): the work behind the
// throughput of k_intersect_df, for comparison with the reference traversal's test counts.
__global__ void __launch_bounds__(kBlock, 8) k_intersect_df_counted(const __grid_constant__ DevScene S,
                                                                 const float* __restrict__ rays, uint32_t n,
                                                                 spt_hit* __restrict__ hits, uint32_t* status,
                                                                 unsigned long long* next,
                                                                 unsigned long long* counts) {
    __shared__ WarpQueue q[kBlock / 32];
    RayBatch<8, false> b{S, rays, nullptr, hits};
    persistent_trace<kWideStack, true>(q[threadIdx.x >> 5], b, n, next, kWideStack, status, counts);
}

template <int TRAV, int STRIDE>
__global__ void __launch_bounds__(kBlock) k_intersect(DevScene S, const float* __restrict__ rays, uint64_t n,
                                                      spt_hit* __restrict__ hits, uint32_t* status) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V3 ro, rd;
    load_ray<STRIDE, false>(rays, i, ro, rd);
    Hit1 h = trace_closest<TRAV>(S, ro, rd, status);
    spt_hit o;
    o.t = h.t;
    o.prim_id = h.found ? slot_prim(S, h.slot) : SPT_MISS;
    o.u = h.u;
    o.v = h.v;
    hits[i] = o;
}

template <int STRIDE, bool FULL>
__global__ void __launch_bounds__(kBlock) k_count(DevScene S, const float* __restrict__ rays, uint64_t n,
                                                  spt_hit* __restrict__ ref_hits, uint32_t* __restrict__ tests,
                                                  uint32_t* __restrict__ nhits, uint32_t* __restrict__ prim_tests,
                                                  uint32_t* status) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V3 ro, rd;
    load_ray<STRIDE, false>(rays, i, ro, rd);
    CountOut c;
    Hit1 h = count_traverse<kStack, FULL>(S, ro, rd, c, status);
    if (FULL && ref_hits) {
        spt_hit o;
        o.t = h.t;
        o.prim_id = h.found ? slot_prim(S, h.slot) : SPT_MISS;
        o.u = h.u;
        o.v = h.v;
        ref_hits[i] = o;
    }
    if (tests) tests[i] = c.tests;
    if (FULL && nhits) nhits[i] = c.hits;
    if (prim_tests) prim_tests[i] = c.prim_tests;
}

// Per-image statistics of integrator.h:47-54, reduced per warp then once per warp to global.
struct StatAcc {
    unsigned long long sum_tests, sum_hits, min_tests, max_tests, min_hits, max_hits;
};

__device__ __forceinline__ void reduce_stats(StatAcc* g, bool valid, uint32_t tests, uint32_t hits) {
    unsigned long long st = valid ? tests : 0ull, sh = valid ? hits : 0ull;
    unsigned mnt = valid ? tests : 0xFFFFFFFFu, mxt = valid ? tests : 0u;
    unsigned mnh = valid ? hits : 0xFFFFFFFFu, mxh = valid ? hits : 0u;
    for (int o = 16; o > 0; o >>= 1) {
        st += __shfl_xor_sync(0xFFFFFFFFu, st, o);
        sh += __shfl_xor_sync(0xFFFFFFFFu, sh, o);
    }
    mnt = __reduce_min_sync(0xFFFFFFFFu, mnt);
    mxt = __reduce_max_sync(0xFFFFFFFFu, mxt);
    mnh = __reduce_min_sync(0xFFFFFFFFu, mnh);
    mxh = __reduce_max_sync(0xFFFFFFFFu, mxh);
    if ((threadIdx.x & 31) == 0 && mnt != 0xFFFFFFFFu) {
        atomicAdd(&g->sum_tests, st);
        atomicAdd(&g->sum_hits, sh);
        atomicMin(&g->min_tests, static_cast<unsigned long long>(mnt));
        atomicMax(&g->max_tests, static_cast<unsigned long long>(mxt));
        atomicMin(&g->min_hits, static_cast<unsigned long long>(mnh));
        atomicMax(&g->max_hits, static_cast<unsigned long long>(mxh));
    }
}

// 256 threads cover a 16x16 pixel tile; each warp an 8x4 sub-tile, so neighbouring lanes trace
// neighbouring pixels (coherent primary rays).
__device__ __forceinline__ void tile_pixel(uint32_t row_stride, uint32_t& x, uint32_t& y) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    x = blockIdx.x * 16 + (w & 1) * 8 + (lane & 7);
    y = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.y) * row_stride % gridDim.y) * 16 + (w >> 1) * 4 + (lane >> 3);
}

// The depth and normal casters over the 8-wide tree: a warp traces its 8x4 pixels together
// (traverse_wide.cuh), and the hit's pixel value goes straight out.  What bounds them is the integer unit
// (64 % of its cycles: permutes, minima and masks of the box tests) and, for a fifth of the time, the longest
// of the grazing rays.  1920x1080 normals of the 1.31M-triangle mesh take 526 us; each lane testing its own
// triangles took 615, the queries' persistent warps, which refill lanes with other tiles' pixels, 618.
template <int MODE>
struct TilePixels {
    const DevScene& S;
    const DevCamera& cam;
    float* out;
    __device__ __forceinline__ void move(uint32_t) {}
    __device__ __forceinline__ const float* root_min() const { return S.root_min; }
    __device__ __forceinline__ const float* root_max() const { return S.root_max; }
    __device__ __forceinline__ WideScene scene() const { return wide_scene(S); }
    __device__ __forceinline__ void store(uint32_t i, float t, uint32_t prim, float u, float v) {
        const bool found = prim != SPT_MISS;
        if (MODE == SPT_RAYCAST_DEPTH) {
            out[i] = found ? t : -1.0f;
            return;
        }
        V3 nrm = v3(0.0f, 0.0f, 0.0f);
        if (found) {
            V3 pos = nrm;   // a sphere's normal needs the hit point: the pixel's ray again
            const Surface sf = surface_of(S, prim);
            if (sf.type == SPT_PRIM_SPHERE) {
                V3 o, d;
                camera_ray(cam, static_cast<float>(i % cam.width) + 0.5f, static_cast<float>(i / cam.width) + 0.5f, o, d);
                pos = hit_pos(true, o, d, t);
            }
            nrm = hit_normal(S, sf, prim, u, v, pos);
        }
        float* q = out + 3ull * i;
        q[0] = nrm.x; q[1] = nrm.y; q[2] = nrm.z;
    }
};

constexpr int kTileBlock = 128;   // 16 x 8 pixels
template <int MODE>
__global__ void __launch_bounds__(kTileBlock, 8) k_raycast_wide(const __grid_constant__ DevScene S,
                                                                const __grid_constant__ DevCamera cam,
                                                                float* __restrict__ out, uint32_t* status) {
    __shared__ WarpQueue wq[kTileBlock / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t x = blockIdx.x * 16 + (w & 1) * 8 + (lane & 7), y = blockIdx.y * 8 + (w >> 1) * 4 + (lane >> 3);
    const bool valid = x < cam.width && y < cam.height;
    V3 o = v3(0.0f, 0.0f, 0.0f), d = o;
    if (valid) camera_ray(cam, static_cast<float>(x) + 0.5f, static_cast<float>(y) + 0.5f, o, d);
    TilePixels<MODE> src{S, cam, out};
    trace_tile<kWideStack>(wq[w], src, valid, o, d, y * cam.width + x, status);
}

// STATS: the image's statistics (tests and passes of the reference's own traversal, which gives the hit
// as well).
// TRAV: the closest-hit traversal without statistics (0 binary, 1 8-wide).
template <int MODE, bool STATS, int TRAV = 0>
__global__ void __launch_bounds__(256) k_raycast(const __grid_constant__ DevScene S, const __grid_constant__ DevCamera cam,
                                                 uint32_t row_stride, void* __restrict__ out, StatAcc* stats,
                                                 uint32_t* status) {
    uint32_t x, y;
    tile_pixel(row_stride, x, y);
    const bool valid = x < cam.width && y < cam.height;
    uint32_t tests = 0, hits = 0;
    if (valid) {
        V3 o, d;
        camera_ray(cam, static_cast<float>(x) + 0.5f, static_cast<float>(y) + 0.5f, o, d);
        const uint64_t idx = static_cast<uint64_t>(y) * cam.width + x;
        if (MODE == SPT_RAYCAST_COUNT && !STATS) {
            CountOut c;
            count_traverse<kStack, false>(S, o, d, c, status);
            static_cast<long long*>(out)[idx] = static_cast<long long>(c.tests);
        } else if (STATS) {
            CountOut c;
            Hit1 h = count_traverse<kStack, true>(S, o, d, c, status);
            tests = c.tests;
            hits = c.hits;
            if (MODE == SPT_RAYCAST_COUNT) {
                static_cast<long long*>(out)[idx] = static_cast<long long>(c.tests);
            } else if (MODE == SPT_RAYCAST_DEPTH) {
                static_cast<float*>(out)[idx] = h.found ? h.t : -1.0f;
            } else {
                V3 nrm = v3(0.0f, 0.0f, 0.0f);
                if (h.found) {
                    const uint32_t prim = slot_prim(S, h.slot);
                    const Surface sf = surface_of(S, prim);
                    nrm = hit_normal(S, sf, prim, h.u, h.v, hit_pos(sf.type == SPT_PRIM_SPHERE, o, d, h.t));
                }
                float* q = static_cast<float*>(out) + 3 * idx;
                q[0] = nrm.x; q[1] = nrm.y; q[2] = nrm.z;
            }
        } else {
            Hit1 h = trace_closest<TRAV>(S, o, d, status);
            if (MODE == SPT_RAYCAST_DEPTH) {
                static_cast<float*>(out)[idx] = h.found ? h.t : -1.0f;
            } else {
                V3 nrm = v3(0.0f, 0.0f, 0.0f);
                if (h.found) {
                    const uint32_t prim = slot_prim(S, h.slot);
                    const Surface sf = surface_of(S, prim);
                    nrm = hit_normal(S, sf, prim, h.u, h.v, hit_pos(sf.type == SPT_PRIM_SPHERE, o, d, h.t));
                }
                float* q = static_cast<float*>(out) + 3 * idx;
                q[0] = nrm.x; q[1] = nrm.y; q[2] = nrm.z;
            }
        }
    }
    if (STATS) reduce_stats(stats, valid, tests, hits);
}

inline unsigned blocks_for(uint64_t n, int block) { return static_cast<unsigned>((n + block - 1) / block); }

}  // namespace

namespace {

// the persistent kernel's grid on the context's device (one computation per context and ray layout)
template <int STRIDE>
int df_grid(spt_context* ctx) {
    int& grid = ctx->df_grid[STRIDE == 6 ? 1 : 0];
    if (!grid) grid = persistent_grid(ctx, reinterpret_cast<const void*>(k_intersect_df<STRIDE>), kBlock);
    return grid;
}

// A caller's traced count held to the batch: *out = min(order[2n], n), so that an order made for
// another batch cannot take the traversal past this one's order entries and hit slots; and the
// persistent kernel's ray counter zeroed, in the same one-thread launch.
__global__ void k_order_count_clamp(const uint32_t* __restrict__ order, uint64_t n, uint32_t* __restrict__ out,
                                    unsigned long long* __restrict__ next) {
    const uint32_t c = order[2 * n];
    *out = c < n ? c : static_cast<uint32_t>(n);
    *next = 0ull;
}

// The persistent closest-hit launch (in the order `order` when it is not NULL, over the count at
// `count`, the hits then in that order; the ordered kernel has the plain one's registers and block,
// so the same grid).
template <int STRIDE>
spt_status launch_df(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n, spt_hit* d_hits,
                     unsigned long long* next, cudaStream_t s, const uint32_t* order = nullptr,
                     const uint32_t* count = nullptr) {
    if (order)
        k_intersect_df_ordered<STRIDE>
            <<<df_grid<STRIDE>(ctx), kBlock, 0, s>>>(sc->dev, d_rays, order, count, d_hits, ctx->d_status, next);
    else
        k_intersect_df<STRIDE><<<df_grid<STRIDE>(ctx), kBlock, 0, s>>>(sc->dev, d_rays, static_cast<uint32_t>(n), d_hits,
                                                                     ctx->d_status, next);
    SPT_CUDA(ctx, cudaGetLastError());
    return SPT_OK;
}

template <int STRIDE>
spt_status launch_intersect_t(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n, spt_hit* d_hits,
                              cudaStream_t s, bool order) {
    if (sc->dev.traversal == 2) {
        unsigned long long* next = nullptr;
        spt_status st = fetch_counter(ctx, s, &next);
        if (st != SPT_OK) return st;
        if (order && n >= order_min_rays() && n <= 0xFFFFFFFFull) {
            // this stream's buffers: the hits in the order first (16-byte aligned for the kernel's
            // float4 stores whatever n is), then the keys (n words), the order, its inverse and the
            // traced count (2n + 1), and the sort's counts
            const size_t work = order_scratch_bytes(ctx);
            void* mem = nullptr;
            if ((st = stream_scratch(ctx, s, (7 * n + 1) * sizeof(uint32_t) + work, &mem)) != SPT_OK) return st;
            if (mem) {
                spt_hit* ordered = static_cast<spt_hit*>(mem);
                uint32_t* keys = reinterpret_cast<uint32_t*>(ordered + n);
                uint32_t* ord = keys + n;
                uint32_t* w = keys + 3 * n + 1;
                if ((st = order_rays(ctx, sc, d_rays, n, STRIDE, s, keys, w, ord)) != SPT_OK) return st;
                if ((st = launch_df<STRIDE>(ctx, sc, d_rays, n, ordered, next, s, ord, ord + 2 * n)) != SPT_OK) return st;
                return unorder_hits(ctx, ordered, ord, n, d_hits, s);
            }
            // every per-stream buffer belongs to another stream: the batch's own order
        }
        // the kernel counts rays in 32 bits: a larger batch goes in runs, each with its own counter
        constexpr uint64_t kRun = 1ull << 31;
        for (uint64_t at = 0; at < n; at += kRun) {
            if (at && (st = fetch_counter(ctx, s, &next)) != SPT_OK) return st;
            if ((st = launch_df<STRIDE>(ctx, sc, d_rays + STRIDE * at, std::min(kRun, n - at), d_hits + at, next, s)) != SPT_OK)
                return st;
        }
        return SPT_OK;
    } else if (sc->dev.traversal == 1) {
        k_intersect<1, STRIDE><<<blocks_for(n, kBlock), kBlock, 0, s>>>(sc->dev, d_rays, n, d_hits, ctx->d_status);
    } else {
        k_intersect<0, STRIDE><<<blocks_for(n, kBlock), kBlock, 0, s>>>(sc->dev, d_rays, n, d_hits, ctx->d_status);
    }
    SPT_CUDA(ctx, cudaGetLastError());
    return SPT_OK;
}

}  // namespace

spt_status launch_intersect(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n, spt_hit* d_hits,
                            cudaStream_t s, int stride, bool order) {
    if (n == 0) return SPT_OK;
    if (n > (1ull << 36)) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "too many rays in one call");
    if (stride == 6) return launch_intersect_t<6>(ctx, sc, d_rays, n, d_hits, s, order);
    return launch_intersect_t<8>(ctx, sc, d_rays, n, d_hits, s, order);
}

// launch_intersect with the persistent kernel's ray counter supplied by the caller (zeroed on stream s
// before this launch) instead of taken from the context's ring, which is allocated on first use.
spt_status launch_intersect_fixed(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                                  spt_hit* d_hits, unsigned long long* next, cudaStream_t s) {
    if (n == 0) return SPT_OK;
    if (sc->dev.traversal != 2) return launch_intersect(ctx, sc, d_rays, n, d_hits, s);  // no counter needed
    return launch_df<8>(ctx, sc, d_rays, n, d_hits, next, s);
}

// k_intersect_df_counted over n rays (8 floats each); counts (device): node visits, primitive tests.
spt_status launch_intersect_counted(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                                   spt_hit* d_hits, unsigned long long* counts, cudaStream_t s) {
    if (n == 0) return SPT_OK;
    if (sc->dev.traversal != 2) return fail(ctx, SPT_ERR_UNSUPPORTED, "the scene has no 8-wide tree");
    unsigned long long* next = nullptr;
    spt_status st = fetch_counter(ctx, s, &next);
    if (st != SPT_OK) return st;
    static_assert(sizeof(unsigned long long) == 8, "");
    constexpr uint64_t kRun = 1ull << 31;   // rays the kernel counts in one launch
    for (uint64_t at = 0; at < n; at += kRun) {
        if (at && (st = fetch_counter(ctx, s, &next)) != SPT_OK) return st;
        k_intersect_df_counted<<<df_grid<8>(ctx), kBlock, 0, s>>>(sc->dev, d_rays + 8 * at,
                                                                static_cast<uint32_t>(std::min(kRun, n - at)), d_hits + at,
                                                                ctx->d_status, next, counts);
    }
    SPT_CUDA(ctx, cudaGetLastError());
    return SPT_OK;
}

spt_status launch_count(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n, spt_hit* d_ref_hits,
                        uint32_t* d_tests, uint32_t* d_hits, uint32_t* d_prim_tests, cudaStream_t s, int stride) {
    if (n == 0) return SPT_OK;
    if (n > (1ull << 36)) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "too many rays in one call");
    // the test counts alone need no primitive tested
    const bool full = d_ref_hits || d_hits;
    auto k = stride == 6 ? (full ? k_count<6, true> : k_count<6, false>) : (full ? k_count<8, true> : k_count<8, false>);
    k<<<blocks_for(n, kBlock), kBlock, 0, s>>>(sc->dev, d_rays, n, d_ref_hits, d_tests, d_hits, d_prim_tests, ctx->d_status);
    SPT_CUDA(ctx, cudaGetLastError());
    return SPT_OK;
}

// The stride of the order in which k_raycast starts the rows of tiles: about 0.618 of their number and
// coprime to it, so every row comes once and neighbours start far apart.  Rows of grazing rays (a
// silhouette's bottom edge), which the counting traversal follows longest, then do not all start last:
// 356 against 370 us for the hit counts at 1277x719.  Normals and depths of small scenes gain too (5,120
// triangles at 1280x720 104 against 115 us); larger ones lose more in L2 than they gain at the end (327,680
// at 1920x1080 421 against 384 us) and take the rows as they come, as the tiled kernel does, which measures
// the same either way.
static uint32_t row_stride(uint32_t rows) {
    uint32_t k = std::max(1u, static_cast<uint32_t>(rows * 0.618));
    auto gcd = [](uint32_t a, uint32_t b) {
        while (b) {
            const uint32_t r = a % b;
            a = b;
            b = r;
        }
        return a;
    };
    while (gcd(k, rows) != 1) ++k;
    return k;
}

static spt_status launch_raycast(spt_context* ctx, const spt_scene* sc, const DevCamera& cam, int32_t mode, void* d_out,
                                 StatAcc* d_stats, cudaStream_t s) {
    dim3 grid((cam.width + 15) / 16, (cam.height + 15) / 16);
    const uint64_t pixels = static_cast<uint64_t>(cam.width) * cam.height;
    const bool wide = sc->dev.traversal >= 1 && !d_stats && mode != SPT_RAYCAST_COUNT;
    // The warp's queue pays once a ray's walk is long, or the image too small to hide a lone thread's latency;
    // in an image of many pixels to a triangle neighbouring rays share their walks.
    // Tiled against one thread per pixel, us a normal image: 1,280 triangles 1920x1080 186 / 142, 640x480 55 / 44; 5,120
    // and 20,480 triangles 1920x1080 227 / 182 and 262 / 225, 320x240 56 / 52 and 60 / 73; 81,920 at 1920x1080 305 /
    // 278, at 640x480 116 / 130; 327,680 at 1600x900 296 / 322, 1920x1080 380 / 383, 2560x1440 593 / 549; 1.31M at
    // 2560x1440 803 / 841, 3840x2160 1,525 / 1,438; 5.24M at 5120x2880 3,859 / 3,955, 7680x4320 7,784 / 7,518.
    const bool short_walks = sc->dev.n_prims <= 2048u || (sc->dev.n_prims <= 131072u && pixels >= 500000u) ||
                             (sc->dev.n_prims > 131072u && pixels >= 6ull * sc->dev.n_prims);
    // the tiled kernel numbers pixels in 32 bits and rows of tiles in 16; larger images (and statistics, the
    // hit counts and scenes without a wide tree) take one thread per pixel
    if (wide && !short_walks && pixels <= 0xFFFFFFFFull && cam.height <= 8u * 65535u) {
        const dim3 tiles((cam.width + 15) / 16, (cam.height + 7) / 8);
        auto k = mode == SPT_RAYCAST_NORMAL ? k_raycast_wide<SPT_RAYCAST_NORMAL> : k_raycast_wide<SPT_RAYCAST_DEPTH>;
        k<<<tiles, kTileBlock, 0, s>>>(sc->dev, cam, static_cast<float*>(d_out), ctx->d_status);
        SPT_CUDA(ctx, cudaGetLastError());
        return SPT_OK;
    }
    auto k = mode == SPT_RAYCAST_NORMAL  ? (d_stats ? k_raycast<SPT_RAYCAST_NORMAL, true> : k_raycast<SPT_RAYCAST_NORMAL, false>)
             : mode == SPT_RAYCAST_DEPTH ? (d_stats ? k_raycast<SPT_RAYCAST_DEPTH, true> : k_raycast<SPT_RAYCAST_DEPTH, false>)
                                         : (d_stats ? k_raycast<SPT_RAYCAST_COUNT, true> : k_raycast<SPT_RAYCAST_COUNT, false>);
    if (wide) k = mode == SPT_RAYCAST_NORMAL ? k_raycast<SPT_RAYCAST_NORMAL, false, 1> : k_raycast<SPT_RAYCAST_DEPTH, false, 1>;
    const bool spread = mode == SPT_RAYCAST_COUNT || d_stats || sc->dev.n_prims <= 32768u;
    k<<<grid, 256, 0, s>>>(sc->dev, cam, spread ? row_stride(grid.y) : 1u, d_out, d_stats, ctx->d_status);
    SPT_CUDA(ctx, cudaGetLastError());
    return SPT_OK;
}

}  // namespace spt

namespace spt {
namespace {

// Rays per pipeline chunk (16 MB in, 8 MB out).  The copy in bounds the pipeline (55 GB/s); what it does not
// hide is the last chunk's query and copy out, and below some size a chunk's query no longer hides behind
// its copy.  3,000,017 rays of 24 bytes take 2.09 / 1.80 / 1.87 ms in chunks of 2^20 / 2^19 / 2^18 rays,
// 2^24 rays 9.31 / 9.08 / 9.36 ms.
constexpr uint64_t kPipeChunk = 1ull << 19;

bool is_pinned(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// Host buffers in page-locked memory: the batch goes through in chunks over the context's pipeline
// streams, chunk c on stream c % kPipe, so the copy in of one chunk, the query of another and the
// copy out of a third run at the same time (PCIe is full duplex).  Each stream owns one set of
// device buffers; its chunks are in stream order, so a set is reused only after its last chunk's
// copy out.
spt_status intersect_pipelined(spt_context* ctx, const spt_scene* sc, const float* rays, uint64_t n, spt_hit* hits,
                               uint32_t* tests, uint32_t* nhits, int stride) {
    const int P = spt_context::kPipe;
    const uint64_t ray_bytes = 4ull * stride;
    const size_t set_bytes = kPipeChunk * (ray_bytes + sizeof(spt_hit) + 4 + 4);
    void* mem;
    spt_status st = scratch(ctx, 9, set_bytes * P, &mem);
    if (st != SPT_OK) return st;
    // the pipeline streams start after whatever the context's stream has queued
    SPT_CUDA(ctx, cudaEventRecord(ctx->ev_pipe[0], ctx->stream));
    for (int i = 0; i < P; ++i) SPT_CUDA(ctx, cudaStreamWaitEvent(ctx->pipe[i], ctx->ev_pipe[0], 0));
    const uint64_t chunks = (n + kPipeChunk - 1) / kPipeChunk;
    for (uint64_t c = 0; c < chunks; ++c) {
        const int i = static_cast<int>(c % P);
        cudaStream_t s = ctx->pipe[i];
        char* base = static_cast<char*>(mem) + set_bytes * i;
        float* d_rays = reinterpret_cast<float*>(base);
        spt_hit* d_hits = reinterpret_cast<spt_hit*>(base + kPipeChunk * ray_bytes);
        uint32_t* d_tests = reinterpret_cast<uint32_t*>(base + kPipeChunk * (ray_bytes + sizeof(spt_hit)));
        uint32_t* d_nh = d_tests + kPipeChunk;
        const uint64_t first = c * kPipeChunk, m = std::min(kPipeChunk, n - first);
        SPT_CUDA(ctx, cudaMemcpyAsync(d_rays, rays + static_cast<uint64_t>(stride) * first, m * ray_bytes,
                                      cudaMemcpyHostToDevice, s));
        if ((st = launch_intersect(ctx, sc, d_rays, m, d_hits, s, stride, true)) != SPT_OK) return st;
        if (tests || nhits)
            if ((st = launch_count(ctx, sc, d_rays, m, nullptr, tests ? d_tests : nullptr, nhits ? d_nh : nullptr,
                                   nullptr, s, stride)) != SPT_OK)
                return st;
        SPT_CUDA(ctx, cudaMemcpyAsync(hits + first, d_hits, m * sizeof(spt_hit), cudaMemcpyDeviceToHost, s));
        if (tests) SPT_CUDA(ctx, cudaMemcpyAsync(tests + first, d_tests, m * 4, cudaMemcpyDeviceToHost, s));
        if (nhits) SPT_CUDA(ctx, cudaMemcpyAsync(nhits + first, d_nh, m * 4, cudaMemcpyDeviceToHost, s));
    }
    // the context's stream continues after every chunk
    for (int i = 0; i < P; ++i) {
        SPT_CUDA(ctx, cudaEventRecord(ctx->ev_pipe[i], ctx->pipe[i]));
        SPT_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->ev_pipe[i], 0));
    }
    return check_status(ctx);
}

// spt_intersect / spt_intersect_packed: stride floats per host ray.
spt_status intersect_host(spt_context* ctx, const spt_scene* sc, const float* rays, uint64_t n, spt_hit* hits,
                          uint32_t* tests, uint32_t* nhits, int stride) {
    if (!ctx || !sc || (n && (!rays || !hits))) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n == 0) return SPT_OK;
    SPT_CUDA(ctx, cudaSetDevice(ctx->device));
    if (n > kPipeChunk && is_pinned(rays) && is_pinned(hits) && (!tests || is_pinned(tests)) &&
        (!nhits || is_pinned(nhits)))
        return intersect_pipelined(ctx, sc, rays, n, hits, tests, nhits, stride);
    spt_status st;
    void *d_rays, *d_hits, *d_tests = nullptr, *d_nh = nullptr;
    const uint64_t ray_bytes = 4ull * stride;
    if ((st = scratch(ctx, 0, n * ray_bytes, &d_rays)) != SPT_OK) return st;
    if ((st = scratch(ctx, 1, n * sizeof(spt_hit), &d_hits)) != SPT_OK) return st;
    if (tests && (st = scratch(ctx, 2, n * 4, &d_tests)) != SPT_OK) return st;
    if (nhits && (st = scratch(ctx, 3, n * 4, &d_nh)) != SPT_OK) return st;
    SPT_CUDA(ctx, cudaMemcpyAsync(d_rays, rays, n * ray_bytes, cudaMemcpyHostToDevice, ctx->stream));
    if ((st = launch_intersect(ctx, sc, static_cast<float*>(d_rays), n, static_cast<spt_hit*>(d_hits), ctx->stream,
                               stride, true)) != SPT_OK)
        return st;
    if (tests || nhits)
        if ((st = launch_count(ctx, sc, static_cast<float*>(d_rays), n, nullptr, static_cast<uint32_t*>(d_tests),
                               static_cast<uint32_t*>(d_nh), nullptr, ctx->stream, stride)) != SPT_OK)
            return st;
    SPT_CUDA(ctx, cudaMemcpyAsync(hits, d_hits, n * sizeof(spt_hit), cudaMemcpyDeviceToHost, ctx->stream));
    if (tests) SPT_CUDA(ctx, cudaMemcpyAsync(tests, d_tests, n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (nhits) SPT_CUDA(ctx, cudaMemcpyAsync(nhits, d_nh, n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    return check_status(ctx);
}

}  // namespace
}  // namespace spt

using namespace spt;

extern "C" {

spt_status spt_intersect(spt_context* ctx, const spt_scene* sc, const float* rays, uint64_t n, spt_hit* hits,
                         uint32_t* tests, uint32_t* nhits) {
    return intersect_host(ctx, sc, rays, n, hits, tests, nhits, 8);
}

spt_status spt_intersect_packed(spt_context* ctx, const spt_scene* sc, const float* rays, uint64_t n, spt_hit* hits,
                                uint32_t* tests, uint32_t* nhits) {
    return intersect_host(ctx, sc, rays, n, hits, tests, nhits, 6);
}

spt_status spt_intersect_device(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                                spt_hit* d_hits, void* stream) {
    if (!ctx || !sc || (n && (!d_rays || !d_hits))) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    return launch_intersect(ctx, sc, d_rays, n, d_hits, static_cast<cudaStream_t>(stream), 8, true);
}

spt_status spt_ray_order_device(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                                uint32_t* d_order, void* stream) {
    if (!ctx || !sc || (n && (!d_rays || !d_order))) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n == 0) return SPT_OK;
    if (n > 0xFFFFFFFFull) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "a ray order holds fewer than 2^32 rays");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    void* mem = nullptr;
    spt_status st = stream_scratch(ctx, s, n * sizeof(uint32_t) + order_scratch_bytes(ctx), &mem);
    if (st != SPT_OK) return st;
    if (!mem) return fail(ctx, SPT_ERR_UNSUPPORTED, "ray order buffers are held by eight other streams");
    uint32_t* keys = static_cast<uint32_t*>(mem);
    return order_rays(ctx, sc, d_rays, n, 8, s, keys, keys + n, d_order);
}

spt_status spt_intersect_ordered_device(spt_context* ctx, const spt_scene* sc, const float* d_rays,
                                        const uint32_t* d_order, uint64_t n, spt_hit* d_hits_ordered, void* stream) {
    if (!ctx || !sc || (n && (!d_rays || !d_order || !d_hits_ordered)))
        return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n == 0) return SPT_OK;
    if (n > 0xFFFFFFFFull) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "a ray order holds fewer than 2^32 rays");
    if (sc->dev.traversal != 2) return fail(ctx, SPT_ERR_UNSUPPORTED, "ordered queries run on the 8-wide persistent traversal");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // two slots of the counter ring: the ray counter and the clamped count, both set by one kernel
    unsigned long long *next = nullptr, *count_slot = nullptr;
    spt_status st = ring_slot(ctx, &next);
    if (st != SPT_OK) return st;
    if ((st = ring_slot(ctx, &count_slot)) != SPT_OK) return st;
    uint32_t* count = reinterpret_cast<uint32_t*>(count_slot);
    k_order_count_clamp<<<1, 1, 0, s>>>(d_order, n, count, next);
    SPT_CUDA(ctx, cudaGetLastError());
    return launch_df<8>(ctx, sc, d_rays, n, d_hits_ordered, next, s, d_order, count);
}

spt_status spt_hits_unorder_device(spt_context* ctx, const uint32_t* d_order, uint64_t n, const spt_hit* d_hits_ordered,
                                   spt_hit* d_hits, void* stream) {
    if (!ctx || (n && (!d_order || !d_hits_ordered || !d_hits))) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (n == 0) return SPT_OK;
    if (n > 0xFFFFFFFFull) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "a ray order holds fewer than 2^32 rays");
    return unorder_hits(ctx, d_hits_ordered, d_order, n, d_hits, static_cast<cudaStream_t>(stream));
}

spt_status spt_traversal_work_device(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                                     spt_hit* d_hits, uint64_t* work) {
    if (!ctx || !sc || !work || (n && (!d_rays || !d_hits)))
        return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    SPT_CUDA(ctx, cudaSetDevice(ctx->device));
    void* d_counts;
    spt_status st = scratch(ctx, 10, 2 * sizeof(unsigned long long), &d_counts);
    if (st != SPT_OK) return st;
    auto* c = static_cast<unsigned long long*>(d_counts);
    SPT_CUDA(ctx, cudaMemsetAsync(c, 0, 2 * sizeof(unsigned long long), ctx->stream));
    if ((st = launch_intersect_counted(ctx, sc, d_rays, n, d_hits, c, ctx->stream)) != SPT_OK) return st;
    unsigned long long h[2] = {0, 0};
    SPT_CUDA(ctx, cudaMemcpyAsync(h, c, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    if ((st = check_status(ctx)) != SPT_OK) return st;   // synchronises the stream
    work[0] = h[0];
    work[1] = h[1];
    return SPT_OK;
}

spt_status spt_count_device(spt_context* ctx, const spt_scene* sc, const float* d_rays, uint64_t n,
                            spt_hit* d_ref_hits, uint32_t* d_tests, uint32_t* d_hits, uint32_t* d_prim_tests,
                            void* stream) {
    if (!ctx || !sc || (n && !d_rays)) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    return launch_count(ctx, sc, d_rays, n, d_ref_hits, d_tests, d_hits, d_prim_tests, static_cast<cudaStream_t>(stream));
}

spt_status spt_raycast_image(spt_context* ctx, const spt_scene* sc, const spt_camera* cam, int32_t mode,
                             void* out_host, spt_render_stats* stats) {
    if (!ctx || !sc || !out_host) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (mode < SPT_RAYCAST_NORMAL || mode > SPT_RAYCAST_COUNT) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "unknown mode");
    SPT_CUDA(ctx, cudaSetDevice(ctx->device));
    DevCamera dc;
    spt_status st = make_camera(ctx, cam, dc);
    if (st != SPT_OK) return st;
    const uint64_t npx = static_cast<uint64_t>(dc.width) * dc.height;
    const size_t elem = mode == SPT_RAYCAST_NORMAL ? 12 : (mode == SPT_RAYCAST_DEPTH ? 4 : 8);
    void *d_out, *d_stats = nullptr;
    if ((st = scratch(ctx, 0, npx * elem, &d_out)) != SPT_OK) return st;
    if (stats) {
        if ((st = scratch(ctx, 4, sizeof(StatAcc), &d_stats)) != SPT_OK) return st;
        StatAcc init{0, 0, std::numeric_limits<unsigned long long>::max(), 0,
                     std::numeric_limits<unsigned long long>::max(), 0};
        SPT_CUDA(ctx, cudaMemcpyAsync(d_stats, &init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
    }
    SPT_CUDA(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    if ((st = launch_raycast(ctx, sc, dc, mode, d_out, static_cast<StatAcc*>(d_stats), ctx->stream)) != SPT_OK) return st;
    SPT_CUDA(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    SPT_CUDA(ctx, cudaMemcpyAsync(out_host, d_out, npx * elem, cudaMemcpyDeviceToHost, ctx->stream));
    StatAcc acc{};
    if (stats) SPT_CUDA(ctx, cudaMemcpyAsync(&acc, d_stats, sizeof(acc), cudaMemcpyDeviceToHost, ctx->stream));
    st = check_status(ctx);
    if (st != SPT_OK) return st;
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->int_tests = acc.sum_tests;
        stats->int_hits = acc.sum_hits;
        stats->min_tests_pp = acc.min_tests;
        stats->max_tests_pp = acc.max_tests;
        stats->min_hits_pp = acc.min_hits;
        stats->max_hits_pp = acc.max_hits;
        stats->paths = npx;
        stats->segments = npx;
        float ms = 0.0f;
        SPT_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
        stats->gpu_ms = ms;
    }
    return SPT_OK;
}

spt_status spt_raycast_image_device(spt_context* ctx, const spt_scene* sc, const spt_camera* cam, int32_t mode,
                                    void* d_out, void* stream) {
    if (!ctx || !sc || !d_out) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "NULL argument");
    if (mode < SPT_RAYCAST_NORMAL || mode > SPT_RAYCAST_COUNT) return fail(ctx, SPT_ERR_INVALID_ARGUMENT, "unknown mode");
    DevCamera dc;
    spt_status st = make_camera(ctx, cam, dc);
    if (st != SPT_OK) return st;
    return launch_raycast(ctx, sc, dc, mode, d_out, nullptr, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
