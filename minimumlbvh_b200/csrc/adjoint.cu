// Differentiable path tracing with a path-replay adjoint (no reference
// counterpart): the gradient of an image loss with respect to per-triangle
// albedo, for the fixed-depth, Russian-roulette-free estimator
//
//   I_p = 1/spp * sum_s L(path_s),   L = sum_{d=0..B} e(t_d) * prod_{j<d} a(t_j)
//
// where t_0 is the primary hit, t_1..t_B the hits after B cosine-sampled
// bounces, e the per-triangle emission and a the per-triangle (grey) albedo.
// Path geometry is that of pt (main_gpu.cu:179-272): Owen-Sobol sample
// streams (dimension 0 for the pixel jitter, 1 + d for bounce d), normals
// facing the incoming ray, origin offset n * 1e-4, Lambertian bounce whose
// cosine/pdf cancels so the throughput is multiplied by the albedo.
//
// The adjoint replays every path from its sample index (paths are never
// stored; Vicini et al., "Path Replay Backpropagation", 2021): with c_d the
// radiance collected at vertex d, dL/da(t_j) = (sum_{d>j} c_d) / a(t_j), and
// grad[t_j] += dLoss/dI_p / spp * that, scattered with atomic adds.
#include <algorithm>

#include "capi_internal.h"
#include "../../include/mlbvh_device.cuh"

namespace mlbvh {

namespace {

// What follows was swept on the differentiation workload (heightfield, 512x512,
// 64 samples, 3 bounces; forward / adjoint ms, start 23.1 / 24.6). Warps per SM
// the kernels are compiled for: 24 19.2 / 19.5, 28 17.9 / 18.2, 32 (64
// registers) 17.2 / 17.2, 40 20.4 / 19.4 (spills). Node visits per round and
// lane: 3 16.9 / 17.5, 4 16.6 / 17.1, 5 16.7 / 16.9, 6 16.8 / 17.1, 8 17.4 /
// 17.4; nodes and leaves in one step, whichever a lane is at: 21.5 / 21.6 (a
// round then pays for both in nearly every step). Lanes that wait before the
// next rays are set up: 8 17.3 / 17.4, 10 16.6 / 17.0, 12 16.6 / 17.1, 16 17.4 /
// 17.4. Leaf tests held back until 8 lanes wait: no gain, 16 lanes: 19.3.
constexpr int kDiffThreads = 64;
constexpr int kDiffWarps = 32;
constexpr int kDiffSteps = 4;
constexpr int kDiffService = 10;
constexpr int kMaxBounces = 8;
constexpr int kDiffStack = 16;       // replay-walk stack entries per lane (shared memory)
constexpr uint32_t kUnit = 64;       // samples per unit of the render's ordered sums; two units are open at a time
constexpr uint32_t kWarpSamples = 512;  // samples a warp takes where the image has enough pixels
constexpr uint32_t kWidePixels = 20000;  // largest image that is shared out by single pixels

struct PathVertex {
    uint32_t tri;
    float collected;  // throughput * emission at this vertex
};

__device__ __forceinline__ Camera camera_of(const mlbvh_ray_generator& g)
{
    Camera c;
    c.origin = mk(g.origin[0], g.origin[1], g.origin[2]);
    c.right = mk(g.right[0], g.right[1], g.right[2]);
    c.up = mk(g.up[0], g.up[1], g.up[2]);
    return c;
}

struct DiffScene {
    int w, h, spp, bounces;
    uint32_t warps, group;  // warps that share the pixels out in groups of so many
    mlbvh_ray_generator gen;
    const mlbvh_node_index* rootPtr;
    const mlbvh_internal_node* nodes;
    const float* tris;
    const float* albedo;
    const float* emission;
};

// The gradient of a path of n vertices, by suffix sums of the collected
// radiance: the part of L that depends on the albedo of vertex j is everything
// collected after it.
__device__ __forceinline__ void scatter(const PathVertex* v, int n, const DiffScene& sc, float g,
                                        float* __restrict__ grad)
{
    float after = 0.0f;
    for (int j = n - 1; j >= 0; --j) {
        if (j < sc.bounces && after != 0.0f) {
            const uint32_t tj = v[j].tri;
            atomicAdd(grad + tj, g * after / __ldg(sc.albedo + tj));
        }
        after += v[j].collected;
    }
}

// Both kernels: a warp traces the samples of its pixels, numbered pixel by
// pixel; its groups of pixels lie all over the image, since neighbouring pixels
// cost alike. Every lane works on a path of its own: it walks
// its ray (intersect_stackfree's closest hit, minimum_lbvh.h:981-1061, through
// the replay walk), and when the ray is done it waits until kDiffService lanes
// do (or as many as still walk); those lanes then shade together, go on with their
// paths' next rays or take the next samples. So a lane whose path ends early
// takes another instead of idling until the warp's longest path is done (with a
// pixel per warp 5.6 of 32 threads were active per instruction, now 15). Bound:
// issue (70 %) and the L1's data stage (76 %).
//
// kAdjoint: the path's vertices are kept and the gradient is scattered when the
// path ends. Otherwise the pixel's radiance is summed in a fixed order,
// whichever lane traced which sample: lane l adds the samples l, l + 32, ... of
// the pixel in turn, and the lanes' sums are added as a pairwise tree in lane
// order, ((p0 + p1) + (p2 + p3)) + ...; the radiances of two units of 64
// samples are kept in shared memory until the older unit is complete.
template <bool kAdjoint>
__device__ __forceinline__ void trace_pixels(const DiffScene& sc, float* __restrict__ image,
                                             float* __restrict__ grad, const float* __restrict__ gradImage)
{
    __shared__ uint2 s_stack[kDiffStack][kDiffThreads];
    __shared__ float s_radiance[kAdjoint ? 1 : kDiffThreads / 32][kAdjoint ? 1 : 2 * kUnit];
    uint2* const stack = &s_stack[0][threadIdx.x];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t pixels = (uint32_t)(sc.w * sc.h), spp = (uint32_t)sc.spp;
    // the warp's pixels: group w, w + warps, ... of the image's; only the image's last group may be partial
    const uint32_t groups = (pixels + sc.group - 1) / sc.group;
    const uint32_t w = blockIdx.x * (kDiffThreads / 32) + warp;
    if (w >= sc.warps) return;
    uint32_t mine = (groups - w + sc.warps - 1) / sc.warps * sc.group;
    if ((groups - 1 - w) % sc.warps == 0) mine -= groups * sc.group - pixels;
    const uint32_t total = mine * spp;
    auto pixel_of = [&](uint32_t i) {  // the warp's i-th
        const uint32_t k = i / sc.group;
        return (k * sc.warps + w - k) * sc.group + i;
    };
    const Camera cam = camera_of(sc.gen);
    const uint32_t root = __ldg(sc.rootPtr);
    float* const radiance = kAdjoint ? nullptr : s_radiance[kAdjoint ? 0 : warp];

    uint32_t next = 0;         // warp-uniform: samples handed out
    uint32_t retired = 0;      // warp-uniform (render): samples summed, in whole units
    uint32_t left0 = kUnit, left1 = kUnit;  // warp-uniform (render): unfinished samples of the open even and odd unit
    float partial = 0.0f;      // render: this lane's sum of the pixel being retired
    // the lane's path: the segment in flight (-1: no path), its sample and state
    int d = -1;
    bool walking = false;
    uint32_t sample = 0, s = 0, xi = 0, yi = 0;
    float throughput = 1.0f, L = 0.0f, g = 0.0f;
    PathVertex v[kAdjoint ? kMaxBounces + 1 : 1];
    f3 ro = mk(0, 0, 0), rd = ro, inv = ro;
    HitRecord hit;
    hit.t = kFltMax;
    hit.tri = 0;
    hit.ng = ro;
    uint32_t curr = 0, prev = 0, steps = 0;
    int depth = 0;
    for (;;) {
        const uint32_t limit = kAdjoint ? total : min(total, retired + 2 * kUnit);
        const int walkers = __popc(__ballot_sync(0xffffffffu, walking));
        const int waiting = __popc(__ballot_sync(0xffffffffu, !walking && (d >= 0 || next < limit)));
        if (walkers == 0 && waiting == 0) break;
        if (waiting >= min(kDiffService, max(walkers, 1))) {
            // ---- shade the hits
            bool start = false, ended = false;
            f3 p = ro, n = ro;
            if (!walking && d >= 0) {
                if (hit.t == kFltMax) {
                    ended = true;
                } else {
                    const uint32_t t = hit.tri;
                    const float collected = throughput * __ldg(sc.emission + t);
                    if (kAdjoint) {
                        v[d].tri = t;
                        v[d].collected = collected;
                    } else {
                        L += collected;
                    }
                    if (d++ == sc.bounces) {
                        ended = true;
                    } else {
                        p = ro + rd * hit.t;
                        n = normalize(hit.ng);
                        if (0.0f < dot(n, rd)) n = -n;
                        throughput = throughput * __ldg(sc.albedo + t);
                        start = true;
                    }
                }
            }
            if (kAdjoint) {
                if (ended) {
                    scatter(v, d, sc, g, grad);
                }
            } else {
                if (ended) radiance[sample % (2 * kUnit)] = L;
                left0 -= __popc(__ballot_sync(0xffffffffu, ended && !(sample & kUnit)));
                left1 -= __popc(__ballot_sync(0xffffffffu, ended && (sample & kUnit)));
                __syncwarp();
                while (retired < next && ((retired & kUnit) ? left1 : left0) == kUnit - min(kUnit, total - retired)) {
                    // a unit is complete: add its samples to their pixels
                    const uint32_t unitEnd = retired + min(kUnit, total - retired);
                    for (uint32_t i = retired; i < unitEnd;) {
                        const uint32_t pix = i / spp, s0 = i - pix * spp, end = min(unitEnd, (pix + 1) * spp);
                        for (uint32_t k = i + ((lane - s0) & 31u); k < end; k += 32)
                            partial += radiance[k % (2 * kUnit)];
                        if (end == (pix + 1) * spp) {
                            float sum = partial;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                            if (lane == 0) image[pixel_of(pix)] = sum / (float)spp;
                            partial = 0.0f;
                        }
                        i = end;
                    }
                    if (retired & kUnit)
                        left1 = kUnit;
                    else
                        left0 = kUnit;
                    retired += kUnit;
                    __syncwarp();
                }
            }
            if (ended) d = -1;
            // ---- lanes without a path take the next samples
            const uint32_t end = kAdjoint ? total : min(total, retired + 2 * kUnit);
            const uint32_t idle = __ballot_sync(0xffffffffu, d < 0);
            const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
            if (d < 0 && next < end && rank < end - next) {
                sample = next + rank;
                const uint32_t pix = sample / spp, pixel = pixel_of(pix);
                s = sample - pix * spp;
                xi = pixel % (uint32_t)sc.w;
                yi = pixel / (uint32_t)sc.w;
                throughput = 1.0f;
                L = 0.0f;
                d = 0;
                start = true;
                if (kAdjoint) {
                    g = __ldg(gradImage + pixel) / (float)sc.spp;
                    if (g == 0.0f) {  // nothing to scatter
                        d = -1;
                        start = false;
                    }
                }
            }
            next = min(next + (uint32_t)__popc(idle), max(end, next));
            // ---- the next rays
            if (start) {
                const float2 r = sobol2d(s, xi, yi, (uint32_t)d);
                if (d == 0) {
                    shoot(cam, ((float)xi + r.x) / (float)sc.w, ((float)yi + r.y) / (float)sc.h, ro, rd);
                } else {
                    f3 xaxis, zaxis;
                    onb(n, xaxis, zaxis);
                    const f3 dl = sample_hemisphere(r.x, r.y);
                    ro = p + n * 0.0001f;
                    rd = xaxis * dl.x + zaxis * dl.z + n * dl.y;
                }
                inv = inv_rd(rd);
                hit.t = kFltMax;
                hit.tri = 0xFFFFFFFFu;
                curr = root;
                prev = kInvalid;
                depth = 0;
                steps = 0;
                walking = true;
            }
        }
        // ---- node visits, then the leaf tests
#pragma unroll
        for (int rep = 0; rep < kDiffSteps; ++rep)
            if (walking && !(curr & kLeafBit) && depth >= 0)
                if (!replay_node<false, kDiffStack>(curr, prev, depth, stack, kDiffThreads, hit.t, sc.nodes, ro, inv,
                                                    0.0f))
                    walking = !replay_pop<false>(curr, depth, stack, kDiffThreads, hit.t);
        const bool test = walking && ((curr & kLeafBit) || depth < 0);
        if (test) {
            uint32_t nv = 0, nt = 0;
            walking = !stackfree_replay_step<false, false, kDiffStack>(curr, prev, depth, stack, kDiffThreads, hit,
                                                                       sc.nodes, sc.tris, ro, rd, inv, 0.0f, nv, nt);
        }
        steps += phase_steps<kDiffSteps>(test);
        if (steps >= kMaxTraversalSteps) walking = false;
    }
}

// Small images of few samples (pixel_warps): a warp per pixel, lane l tracing
// the samples l, l + 32, ... in turn, a step of either kind at a time. Nearly
// every path has a warp to itself, so nothing is gained by taking up another,
// and waiting only adds to its chain of loads.
template <bool kAdjoint>
__device__ __forceinline__ void trace_pixel(const DiffScene& sc, float* __restrict__ image, float* __restrict__ grad,
                                            const float* __restrict__ gradImage)
{
    __shared__ uint2 s_stack[kDiffStack][32];
    uint2* const stack = &s_stack[0][threadIdx.x];
    const uint32_t lane = threadIdx.x, pixel = blockIdx.x;
    const uint32_t xi = pixel % (uint32_t)sc.w, yi = pixel / (uint32_t)sc.w;
    const float g = kAdjoint ? __ldg(gradImage + pixel) / (float)sc.spp : 0.0f;
    if (kAdjoint && g == 0.0f) return;  // nothing to scatter
    const Camera cam = camera_of(sc.gen);
    const uint32_t root = __ldg(sc.rootPtr);
    PathVertex v[kAdjoint ? kMaxBounces + 1 : 1];
    float sum = 0.0f;
    for (uint32_t s = lane; s < (uint32_t)sc.spp; s += 32) {
        float throughput = 1.0f, L = 0.0f;
        f3 ro, rd;
        const float2 jitter = sobol2d(s, xi, yi, 0u);
        shoot(cam, ((float)xi + jitter.x) / (float)sc.w, ((float)yi + jitter.y) / (float)sc.h, ro, rd);
        int d = 0;
        for (;;) {
            HitRecord hit;
            hit.t = kFltMax;
            hit.tri = 0xFFFFFFFFu;
            const f3 inv = inv_rd(rd);
            uint32_t curr = root, prev = kInvalid, nv = 0, nt = 0;
            int depth = 0;
            for (uint32_t steps = 1; steps < kMaxTraversalSteps; ++steps)
                if (stackfree_replay_step<false, false, kDiffStack>(curr, prev, depth, stack, 32, hit, sc.nodes, sc.tris,
                                                                    ro, rd, inv, 0.0f, nv, nt))
                    break;
            if (hit.t == kFltMax) break;
            const uint32_t t = hit.tri;
            const float collected = throughput * __ldg(sc.emission + t);
            if (kAdjoint) {
                v[d].tri = t;
                v[d].collected = collected;
            } else {
                L += collected;
            }
            if (d++ == sc.bounces) break;
            const f3 p = ro + rd * hit.t;
            f3 n = normalize(hit.ng);
            if (0.0f < dot(n, rd)) n = -n;
            throughput = throughput * __ldg(sc.albedo + t);
            const float2 r = sobol2d(s, xi, yi, (uint32_t)d);
            f3 xaxis, zaxis;
            onb(n, xaxis, zaxis);
            const f3 dl = sample_hemisphere(r.x, r.y);
            ro = p + n * 0.0001f;
            rd = xaxis * dl.x + zaxis * dl.z + n * dl.y;
        }
        if (kAdjoint)
            scatter(v, d, sc, g, grad);
        else
            sum += L;
    }
    if (!kAdjoint) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) image[pixel] = sum / (float)sc.spp;
    }
}
__global__ void __launch_bounds__(32, 24) k_pt_diff_render_pixel(float* __restrict__ image, DiffScene sc)
{
    trace_pixel<false>(sc, image, nullptr, nullptr);
}
__global__ void __launch_bounds__(32, 24)
    k_pt_diff_adjoint_pixel(float* __restrict__ grad, const float* __restrict__ gradImage, DiffScene sc)
{
    trace_pixel<true>(sc, nullptr, grad, gradImage);
}

__global__ void __launch_bounds__(kDiffThreads, kDiffWarps * 32 / kDiffThreads)
    k_pt_diff_render(float* __restrict__ image, DiffScene sc)
{
    trace_pixels<false>(sc, image, nullptr, nullptr);
}

__global__ void __launch_bounds__(kDiffThreads, kDiffWarps * 32 / kDiffThreads)
    k_pt_diff_adjoint(float* __restrict__ grad, const float* __restrict__ gradImage, DiffScene sc)
{
    trace_pixels<true>(sc, nullptr, grad, gradImage);
}

// Views 2.5 times as wide as high and more: their long paths lie in a few
// columns, the others end at once.
bool is_wide(const DiffScene& sc) { return 2ll * sc.w >= 5ll * sc.h; }

// The warps and their groups of pixels. A warp takes kWarpSamples samples at
// most, four rounds of resident warps where that leaves it 128 samples, else two;
// below 32, 32 samples (a warp's lanes share its instructions) as long as 16 warps
// per SM remain: few samples finish soonest spread out. A group is as many pixels
// as 32 samples need, so that the lanes trace neighbouring rays, or all of the
// warp's where it has less than two such groups; a single pixel where its samples
// nearly fill the warp, or half of it in a wide view, and in small wide views. A
// warp's samples stay below 2^31. Render and adjoint, 3 bounces, 213,000-triangle
// heightfield, us, with consecutive pixels in a warp / with groups all over the
// image: 512x32, 32 samples 830 / 550; 400x60, 64 2,308 / 1,303; 1024x128, 32 4,987 /
// 2,260; 512x512, 64 35,500 / 34,100, 4 2,969 / 2,925. 180 images drawn over 32 to 512
// pixels a side, 1 to 64 samples, 1 to 3 bounces: 1.08x on average, 0.945x to 1.6x.
void share_out(DiffScene& sc)
{
    using u64 = unsigned long long;
    const u64 w = (u64)sc.w, pixels = w * sc.h, spp = (u64)sc.spp, samples = pixels * spp;
    const uint32_t sms = (uint32_t)device_sm_count();
    const u64 round = samples / (kDiffWarps * sms);
    u64 k = std::min<u64>(std::max(round / 4, std::min<u64>(round / 2, 128)), kWarpSamples);
    const bool few = k < 32;
    if (few) k = std::max<u64>(1, std::min<u64>(32, samples / (16u * sms)));
    const bool single = spp >= (is_wide(sc) ? 16 : 24) || (few && is_wide(sc) && pixels <= kWidePixels);
    const u64 lanes = k < 64 ? k : 32;  // samples of a group
    const u64 group = single ? 1 : (lanes + spp - 1) / spp, groups = (pixels + group - 1) / group;
    const u64 per = std::max<u64>(1, k / (group * spp));  // groups of a warp
    u64 warps = (groups + per - 1) / per;
    // a warp's next group lies 0.38 of a row further on: never in the same columns
    if (per > 1) warps += (w * 382 / 1000 + w - warps * group % w) % w / group;
    sc.group = (uint32_t)group;
    sc.warps = (uint32_t)std::min(warps, groups);
}

// A warp per pixel (trace_pixel): small images of few samples, wide ones up to
// 16,000 pixels and 16 samples. Render and adjoint, 3 bounces, against the warps
// above, us: 32x32 at 1 / 4 / 8 / 16 samples 216 / 317 / 380 / 464 against 241 / 340 / 386 /
// 472, 64x64 269 / 366 / 452 / 572 against 311 / 404 / 501 / 555, 80x80 314 / 503 / 654 / 833
// against 323 / 463 / 525 / 591; 300x40 at 4 samples 348 against 388.
bool pixel_warps(const DiffScene& sc)
{
    const uint32_t pixels = (uint32_t)sc.w * (uint32_t)sc.h, spp = (uint32_t)sc.spp, sms = (uint32_t)device_sm_count();
    if (is_wide(sc)) return spp <= 16 && pixels <= 108 * sms;
    return spp <= 12 && pixels <= 52 * sms && pixels * spp <= 256 * sms;
}
uint32_t diff_blocks(const DiffScene& sc) { return (sc.warps + kDiffThreads / 32 - 1) / (kDiffThreads / 32); }

mlbvh_status check_diff_args(int w, int h, int spp, int bounces, const void* a, const void* b, const void* c,
                             const void* d, const void* e)
{
    if (w <= 0 || h <= 0 || (long long)w * h >= (1ll << 31)) return fail(MLBVH_ERR_INVALID_ARG, "bad image size");
    if (spp <= 0) return fail(MLBVH_ERR_INVALID_ARG, "spp must be positive");
    if (bounces < 0 || bounces > kMaxBounces) return fail(MLBVH_ERR_INVALID_ARG, "bounces must be in [0, 8]");
    if (!a || !b || !c || !d || !e) return fail(MLBVH_ERR_INVALID_ARG, "null pointer");
    if (!aligned16(a) || !aligned16(b) || !aligned16(c) || !aligned16(d) || !aligned16(e))
        return fail(MLBVH_ERR_INVALID_ARG, "device pointers must be 16-byte aligned");
    return MLBVH_OK;
}

}  // namespace

mlbvh_status pt_diff_render(float* dImage, int w, int h, int spp, int bounces, const mlbvh_ray_generator& cam,
                            const mlbvh_node_index* dRoot, const mlbvh_internal_node* dNodes,
                            const mlbvh_triangle* dTris, const float* dAlbedo, const float* dEmission,
                            cudaStream_t stream)
{
    if (mlbvh_status s = check_diff_args(w, h, spp, bounces, dImage, dRoot, dTris, dAlbedo, dEmission)) return s;
    if (!aligned32(dNodes)) return fail(MLBVH_ERR_INVALID_ARG, "device pointers must be 16-byte aligned");
    if ((long long)w * h * 32 >= (1ll << 31)) return fail(MLBVH_ERR_INVALID_ARG, "bad image size");
    DiffScene sc{w, h, spp, bounces, 0, 0, cam, dRoot, dNodes, reinterpret_cast<const float*>(dTris), dAlbedo,
                 dEmission};
    if (pixel_warps(sc)) {
        k_pt_diff_render_pixel<<<(unsigned)(w * h), 32, 0, stream>>>(dImage, sc);
    } else {
        share_out(sc);
        k_pt_diff_render<<<diff_blocks(sc), kDiffThreads, 0, stream>>>(dImage, sc);
    }
    MLBVH_CHECK_LAUNCH("k_pt_diff_render");
    return MLBVH_OK;
}

mlbvh_status pt_diff_adjoint(float* dGrad, const float* dGradImage, int w, int h, int spp, int bounces,
                             const mlbvh_ray_generator& cam, const mlbvh_node_index* dRoot,
                             const mlbvh_internal_node* dNodes, const mlbvh_triangle* dTris, const float* dAlbedo,
                             const float* dEmission, cudaStream_t stream)
{
    if (mlbvh_status s = check_diff_args(w, h, spp, bounces, dGrad, dRoot, dTris, dAlbedo, dEmission)) return s;
    if (!dGradImage || !aligned16(dGradImage) || !aligned32(dNodes))
        return fail(MLBVH_ERR_INVALID_ARG, "null or misaligned pointer");
    if ((long long)w * h * 32 >= (1ll << 31)) return fail(MLBVH_ERR_INVALID_ARG, "bad image size");
    DiffScene sc{w, h, spp, bounces, 0, 0, cam, dRoot, dNodes, reinterpret_cast<const float*>(dTris), dAlbedo,
                 dEmission};
    if (pixel_warps(sc)) {
        k_pt_diff_adjoint_pixel<<<(unsigned)(w * h), 32, 0, stream>>>(dGrad, dGradImage, sc);
    } else {
        share_out(sc);
        k_pt_diff_adjoint<<<diff_blocks(sc), kDiffThreads, 0, stream>>>(dGrad, dGradImage, sc);
    }
    MLBVH_CHECK_LAUNCH("k_pt_diff_adjoint");
    return MLBVH_OK;
}

}  // namespace mlbvh
