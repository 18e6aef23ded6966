// The ray queries' common schedules. The pool: a CTA takes blocks of 32
// consecutive rays from all over the array, and a lane whose ray is done takes
// the CTA's next ray. Or one ray per thread.
#pragma once

#include <algorithm>
#include <cstdint>

#include "../../include/mlbvh_device.cuh"

namespace mlbvh {

// One ray per thread left a warp's lanes idle until its longest ray was done.
// Measured (B200; 1M random rays over the 213k-triangle heightfield, closest
// hit, one ray per thread / pool): binary tree 450 / 326 us, 4-wide 431 / 328,
// quantised 4-wide 453 / 342, quantised binary 519 / 366; 1M camera rays over
// the 4M-triangle soup: 485 / 447, 430 / 373, 523 / 437, 544 / 510. Swept:
// CTAs of 64 threads up to 20 % slower, two waves of CTAs 15 %, contiguous
// chunks per warp 70 % on the camera rays (neighbours cost alike) and within 5 %
// on the random ones; a batch of 4 or 12 within 3 %.
constexpr int kPoolThreads = 128;
constexpr int kPoolBatch = 8;        // lanes that wait for a ray before the next ones are loaded
constexpr uint32_t kMinShift = 3;    // smallest block: 8 rays
constexpr uint32_t kFewLanes = 16;   // below, a warp's round is kFew rounds of node visits long

// The pool of a query of n rays: one CTA per block of 32 rays (fewer rays where
// that leaves multiprocessors idle), as many CTAs as are resident at most; block
// b goes to CTA b modulo their number, so that neighbouring rays, which cost
// alike, are spread over all CTAs. Where the CTA has fewer rays than lanes, its
// warps share them out.
struct RayPool {
    uint32_t n, ctas, lanes, shift;  // rays, CTAs, lanes used of each warp, log2 of the block
};
// warps: resident warps per SM of the kernel.
inline RayPool ray_pool(uint32_t n, int sms, int warps)
{
    RayPool p{n, 0, 32, 5};
    while (p.shift > kMinShift && (n >> p.shift) < 2u * (uint32_t)sms) --p.shift;
    const uint32_t blocks = (uint32_t)(((uint64_t)n + (1u << p.shift) - 1) >> p.shift);
    p.ctas = std::min(blocks, (uint32_t)sms * (uint32_t)(warps * 32 / kPoolThreads));
    const uint32_t perCta = (blocks + p.ctas - 1) / p.ctas << p.shift, ctaWarps = kPoolThreads / 32;
    p.lanes = std::min(32u, (perCta + ctaWarps - 1) / ctaWarps);
    return p;
}

// Launches of some thousands of rays up to about as many as are resident at once
// run one ray per thread instead, a step of either kind at a time. Latency
// bounds them: a refill has nothing to add where every ray is resident, waiting
// for the warp's node visits only lengthens a ray's chain, and without the
// pool's state more warps fit. Smaller ones stay with the pool, which shares
// their rays out over more warps and multiprocessors. The lines lie where the
// two are even; each kernel has its own. Pool / one ray per thread, us, random
// rays over a 46,000-triangle heightfield (a 1M-triangle soup):
//                     33,000             60,000             130,000
//   binary any        50 / 39 (74 / 68)  49 / 41 (92 / 80)  58 / 47 (128 / 99)
//   binary closest    71 / 64 (135/118)  75 / 70 (150/130)  86 / 79 (179 / 178)
//   4-wide any        42 / 31 (64 / 56)  45 / 33 (75 / 60)  51 / 45 (102 / 81)
//   quantised 4-wide  43 / 33 (62 / 53)  46 / 33 (75 / 62)  54 / 48 (102 / 84)
// and beyond, for 4-wide any hit: 170,000 50 / 48 (94 / 92), 210,000 55 / 54 (99
// / 104), 320,000 69 / 75 (121 / 139). Coherent rays keep an advantage of 5 to 20
// % without the pool up to about 500,000 any-hit rays; random ones lose as much.
constexpr int kEachThreads = 64;
struct EachRange {
    uint32_t from, to;  // rays per multiprocessor
    bool has(uint32_t n, int sms) const { return n >= from * (uint32_t)sms && n <= to * (uint32_t)sms; }
};
template <bool kEach>
constexpr int kRayThreads = kEach ? kEachThreads : kPoolThreads;
inline uint32_t ray_ctas(const RayPool& p, bool each)
{
    return each ? (uint32_t)(((uint64_t)p.n + kEachThreads - 1) / kEachThreads) : p.ctas;
}

// Traces the CTA's rays, kEach: one per thread. start(i, a, b) begins ray i
// ({ro, tmin} {rd, tmax}) and sets the walk's state (curr, depth, hit); step() makes one step and
// returns true when the walk is over; finish(i) follows the ray's Hit record.
// apart(): the lane walks by other rules (a full stack's fallback), nodes and
// leaves alike, and is stepped on its own.
// Up to kNodes node visits alternate with one leaf test (see walk_phases), kFew
// times as many where the warp uses few lanes.
template <bool kEach, int kNodes, int kFew, class Start, class Apart, class Step, class Finish>
__device__ __forceinline__ void trace_rays(const float4* __restrict__ rays, float4* __restrict__ hits, RayPool pool,
                                           const HitRecord& hit, const uint32_t& curr, Start start, Apart apart, Step step,
                                           Finish finish)
{
    if constexpr (kEach) {
        const uint32_t ray = blockIdx.x * kEachThreads + threadIdx.x;
        if (ray >= pool.n) return;
        start(ray, __ldg(rays + 2 * (size_t)ray), __ldg(rays + 2 * (size_t)ray + 1));
        for (uint32_t steps = 1; steps < kMaxTraversalSteps; ++steps)
            if (step()) break;
        hits[2 * (size_t)ray] = make_float4(hit.t, 0.0f, hit.u, hit.v);
        hits[2 * (size_t)ray + 1] = make_float4(hit.ng.x, hit.ng.y, hit.ng.z, __uint_as_float(hit.tri));
        finish(ray);
        return;
    }
    __shared__ uint32_t s_next;
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    // the CTA's rays, block after block; the array's last block may be partial
    const uint32_t size = 1u << pool.shift, blocks = (uint32_t)(((uint64_t)pool.n + size - 1) >> pool.shift);
    const uint32_t mine = (blocks - blockIdx.x + pool.ctas - 1) / pool.ctas << pool.shift;
    const bool used = lane < pool.lanes;
    bool live = false, more = true;  // more: warp-uniform
    const int rounds = pool.lanes < kFewLanes ? kFew : 1;
    uint32_t ray = 0, steps = 0;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, used && !live);
        const uint32_t walkers = __ballot_sync(0xffffffffu, live);
        if (more && idle && (walkers == 0u || __popc(idle) >= kPoolBatch)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&s_next, (uint32_t)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            more = base + __popc(idle) < mine;
            const uint32_t j = base + __popc(idle & ((1u << lane) - 1u));
            if (used && !live && j < mine) {
                ray = (((j >> pool.shift) * pool.ctas + blockIdx.x) << pool.shift) + (j & (size - 1));
                if (ray < pool.n) {
                    start(ray, __ldg(rays + 2 * (size_t)ray), __ldg(rays + 2 * (size_t)ray + 1));
                    steps = 0;
                    live = true;
                }
            }
        } else if (walkers == 0u) {
            return;
        }
        bool done = false;
#pragma unroll 1
        for (int r = 0; r < rounds; ++r) {
#pragma unroll
            for (int k = 0; k < kNodes; ++k)
                if (live && !done && !apart() && !(curr & kLeafBit)) done = step();
        }
        // the fewest steps that the round can hold (phase_steps): the leaf test, or all node visits; as many apart
        steps += (uint32_t)kNodes - (curr >> 31) * (uint32_t)(kNodes - 1);
        if (live && !done && !apart() && (curr & kLeafBit)) done = step();
        if (live && !done && apart()) {  // as many steps of either kind
#pragma unroll 1
            for (int k = 0; k <= kNodes && !done; ++k) done = step();
        }
        if (live && (done || steps >= kMaxTraversalSteps)) {
            hits[2 * (size_t)ray] = make_float4(hit.t, 0.0f, hit.u, hit.v);
            hits[2 * (size_t)ray + 1] = make_float4(hit.ng.x, hit.ng.y, hit.ng.z, __uint_as_float(hit.tri));
            finish(ray);
            live = false;
        }
    }
}

}  // namespace mlbvh
