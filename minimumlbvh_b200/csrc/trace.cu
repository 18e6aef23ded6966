// Ray queries over the reference node layout.
//
// Replaces the per-ray device calls of intersect_stackfree (minimum_lbvh.h:
// 981-1061), intersect_escape_link (:1063-1137) and intersect_stackfull
// (:912-973) with a single launch. MLBVH_TRAVERSAL_STACKFREE and
// MLBVH_TRAVERSAL_REPLAY both run the replay walk, which returns
// intersect_stackfree's Hit records bit for bit and loads every node once
// instead of up to three times (one ray per thread, 1M camera rays of a
// 4M-triangle soup: 0.690 -> 0.505 ms), scheduled by ray_pool.cuh. Rays and
// hits move as 2 x 16-byte vectors, nodes as 2 x 32-byte read-only loads.
#include "capi_internal.h"
#include "../../include/mlbvh_device.cuh"
#include "ray_pool.cuh"

namespace mlbvh {

namespace {

constexpr int kNodeSteps = 4;  // node visits per leaf test (2-4 within 4 %)
constexpr int kPoolWarps = 32;  // resident warps per SM of the pooled trace kernel (64 registers)

constexpr int kEachWarps = 36;  // one ray per thread (56 registers)
// rays per SM that run one per thread: to one and a quarter times the resident ones, any hit; to the resident ones
template <bool kAny>
constexpr EachRange kEachRange = kAny ? EachRange{32, 1440} : EachRange{96, 1152};

constexpr int kFewRounds = 3;  // (257 to 4,000 rays: 1M soup 3 to 7 % faster than 1, heightfield 0 to 6 % slower)

constexpr int kTraceThreads = 64;  // of the one-ray-per-thread walks

constexpr int kReplayDepth = 16;  // stack entries per ray of the replay walk

// intersect_stackfree's Hit records through the replay walk.
template <bool kAny, bool kEach>
__global__ void __launch_bounds__(kRayThreads<kEach>, (kEach ? kEachWarps : kPoolWarps) * 32 / kRayThreads<kEach>)
    k_trace_replay(const mlbvh_internal_node* __restrict__ nodes, const mlbvh_node_index* __restrict__ rootPtr,
                   const float* __restrict__ tris, const float4* __restrict__ rays, float4* __restrict__ hits,
                   RayPool pool)
{
    __shared__ typename ReplayStack<kAny>::Entry s_stack[kReplayDepth][kRayThreads<kEach>];
    const uint32_t root = __ldg(rootPtr);
    f3 ro = mk(0, 0, 0), rd = ro, inv = ro;
    float tmin = 0.0f;
    HitRecord hit;
    uint32_t curr = root, prev = kInvalid, nv = 0, nt = 0;
    int depth = 0;
    trace_rays<kEach, kNodeSteps, kFewRounds>(
        rays, hits, pool, hit, curr,
        [&](uint32_t, float4 a, float4 b) {
            ro = mk(a.x, a.y, a.z);
            rd = mk(b.x, b.y, b.z);
            inv = inv_rd(rd);
            tmin = a.w;
            hit = HitRecord{b.w, 0.0f, 0.0f, mk(0.0f, 0.0f, 0.0f), 0xFFFFFFFFu};
            curr = root;
            prev = kInvalid;
            depth = 0;
        },
        [&] { return depth < 0; },
        [&] {
            return stackfree_replay_step<kAny, false, kReplayDepth>(curr, prev, depth, &s_stack[0][threadIdx.x],
                                                                    kRayThreads<kEach>, hit, nodes, tris, ro, rd, inv, tmin,
                                                                    nv, nt);
        },
        [](uint32_t) {});
}

// The reference's other walks, one ray per thread.
template <int kMode, bool kAny>
__global__ void __launch_bounds__(kTraceThreads)
    k_trace(const mlbvh_internal_node* __restrict__ nodes, const mlbvh_node_index* __restrict__ rootPtr,
            const float* __restrict__ tris, const float4* __restrict__ rays, float4* __restrict__ hits, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = __ldg(rays + 2 * (size_t)i), b = __ldg(rays + 2 * (size_t)i + 1);
    const f3 ro = mk(a.x, a.y, a.z), rd = mk(b.x, b.y, b.z);
    const float tmin = a.w;
    HitRecord hit;
    hit.t = b.w;
    hit.u = 0.0f;
    hit.v = 0.0f;
    hit.ng = mk(0.0f, 0.0f, 0.0f);
    hit.tri = 0xFFFFFFFFu;
    const uint32_t root = __ldg(rootPtr);
    const f3 inv = inv_rd(rd);
    if (kMode == MLBVH_TRAVERSAL_ESCAPE_LINK) {
        trace_escape<kAny>(hit, nodes, tris, root, ro, rd, inv, tmin);
    } else {
        uint32_t stack[64];
        trace_stackfull(hit, nodes, tris, root, ro, rd, inv, tmin, stack, 64);
    }
    hits[2 * (size_t)i] = make_float4(hit.t, 0.0f, hit.u, hit.v);
    hits[2 * (size_t)i + 1] = make_float4(hit.ng.x, hit.ng.y, hit.ng.z, __uint_as_float(hit.tri));
}

}  // namespace

mlbvh_status trace(const mlbvh_internal_node* dNodes, const mlbvh_node_index* dRoot, const mlbvh_triangle* dTris,
                   const mlbvh_ray* dRays, mlbvh_hit* dHits, uint32_t nRays, int rayQuery, int traversal,
                   cudaStream_t stream)
{
    if (nRays == 0) return MLBVH_OK;
    if (!dRoot || !dTris || !dRays || !dHits) return fail(MLBVH_ERR_INVALID_ARG, "null pointer");
    if (!aligned32(dNodes) || !aligned16(dRoot) || !aligned16(dTris) || !aligned16(dRays) || !aligned16(dHits))
        return fail(MLBVH_ERR_INVALID_ARG, "device pointers must be 16-byte aligned (node arrays 32-byte)");
    if (rayQuery != MLBVH_RAY_QUERY_CLOSEST && rayQuery != MLBVH_RAY_QUERY_ANY)
        return fail(MLBVH_ERR_INVALID_ARG, "rayQuery must be MLBVH_RAY_QUERY_CLOSEST or MLBVH_RAY_QUERY_ANY");
    const bool any = rayQuery == MLBVH_RAY_QUERY_ANY;
    const unsigned blocks = (nRays + kTraceThreads - 1) / kTraceThreads;
    const float* tris = reinterpret_cast<const float*>(dTris);
    const float4* rays = reinterpret_cast<const float4*>(dRays);
    float4* hits = reinterpret_cast<float4*>(dHits);
    switch (traversal) {
    case MLBVH_TRAVERSAL_ESCAPE_LINK:
        if (any)
            k_trace<MLBVH_TRAVERSAL_ESCAPE_LINK, true><<<blocks, kTraceThreads, 0, stream>>>(dNodes, dRoot, tris, rays, hits, nRays);
        else
            k_trace<MLBVH_TRAVERSAL_ESCAPE_LINK, false><<<blocks, kTraceThreads, 0, stream>>>(dNodes, dRoot, tris, rays, hits, nRays);
        break;
    case MLBVH_TRAVERSAL_STACKFREE:  // the replay walk's Hit records are the stack-free walk's
    case MLBVH_TRAVERSAL_REPLAY: {
        const RayPool pool = ray_pool(nRays, device_sm_count(), kPoolWarps);
        const bool each = (any ? kEachRange<true> : kEachRange<false>).has(nRays, device_sm_count());
        const auto kernel = any ? (each ? k_trace_replay<true, true> : k_trace_replay<true, false>)
                                : (each ? k_trace_replay<false, true> : k_trace_replay<false, false>);
        kernel<<<ray_ctas(pool, each), each ? kEachThreads : kPoolThreads, 0, stream>>>(dNodes, dRoot, tris, rays, hits,
                                                                                      pool);
        break;
    }
    case MLBVH_TRAVERSAL_STACKFULL:
        k_trace<MLBVH_TRAVERSAL_STACKFULL, false><<<blocks, kTraceThreads, 0, stream>>>(dNodes, dRoot, tris, rays, hits, nRays);
        break;
    default:
        return fail(MLBVH_ERR_INVALID_ARG, "unknown traversal");
    }
    MLBVH_CHECK_LAUNCH("k_trace");
    return MLBVH_OK;
}

}  // namespace mlbvh
