// The ray queries' common schedule: a CTA takes blocks of 32 consecutive rays
// from all over the array, and a lane whose ray is done takes the CTA's next
// ray.
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
constexpr uint32_t kFewLanes = 16;   // below, a warp's round is kFewRounds rounds of node visits long
constexpr int kFewRounds = 3;        // (4,099 rays: 52 us with one round, 49 with three; 4-wide 38 and 36)

// The launch of a query of n rays: one CTA per block of 32 rays (fewer where
// that leaves multiprocessors idle), as many CTAs as are resident at most; block b goes to CTA b modulo their number, so that
// neighbouring rays, which cost alike, are spread over all CTAs. Where the CTA
// has fewer rays than lanes, its warps share them out.
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

// Traces the CTA's rays. start(i, a, b) begins ray i ({ro, tmin} {rd, tmax})
// and sets the walk's state (curr, depth, hit); step() makes one step and
// returns true when the walk is over; finish(i) follows the ray's Hit record.
// apart(): the lane walks by other rules (a full stack's fallback), nodes and
// leaves alike, and is stepped on its own.
// Up to kNodes node visits alternate with one leaf test (see walk_phases).
template <int kNodes, class Start, class Apart, class Step, class Finish>
__device__ __forceinline__ void trace_pool(const float4* __restrict__ rays, float4* __restrict__ hits, RayPool pool,
                                           const HitRecord& hit, const uint32_t& curr, Start start, Apart apart, Step step,
                                           Finish finish)
{
    __shared__ uint32_t s_next;
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    // the CTA's rays, block after block; the array's last block may be partial
    const uint32_t size = 1u << pool.shift, blocks = (uint32_t)(((uint64_t)pool.n + size - 1) >> pool.shift);
    const uint32_t mine = (blocks - blockIdx.x + pool.ctas - 1) / pool.ctas << pool.shift;
    const bool used = lane < pool.lanes;
    bool live = false, more = true;  // more: warp-uniform
    const int rounds = pool.lanes < kFewLanes ? kFewRounds : 1;
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
        const bool test = live && !done && !apart() && (curr & kLeafBit);
        if (test) done = step();
        if (live && !done && apart()) {  // as many steps of either kind
#pragma unroll 1
            for (int k = 0; k <= kNodes && !done; ++k) done = step();
        }
        steps += phase_steps<kNodes>(test);
        if (live && (done || steps >= kMaxTraversalSteps)) {
            hits[2 * (size_t)ray] = make_float4(hit.t, 0.0f, hit.u, hit.v);
            hits[2 * (size_t)ray + 1] = make_float4(hit.ng.x, hit.ng.y, hit.ng.z, __uint_as_float(hit.tri));
            finish(ray);
            live = false;
        }
    }
}

}  // namespace mlbvh
