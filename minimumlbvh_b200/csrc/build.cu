// LBVH build on B200: scene bounds, Morton keys + digit histograms, a
// stable Onesweep LSD radix sort, and the agglomerative bottom-up build.
//
// Replaces BVHGPUBuilder::build (minimum_lbvh.h:783-871), its kernels
// (minimum_lbvh.cu:38-120) and OnesweepSort (tinyhiponesweep.h:592-668).
//
// Launch chain on one stream (no host synchronisation; up to 4,096 triangles
// k_small_sort stands for the first three rows):
//   k_scene_bounds   per-CTA partial bounds of all vertices; zeroes the
//                    sort's counters, histograms and look-back words
//   k_keys           reduces the partial bounds, writes the 32-bit Morton key
//                    of every triangle and accumulates the four 8-bit digit
//                    histograms; resets the build's hand-off words
//   k_onesweep x4    one stable pass per digit: warp multisplit, decoupled
//                    look-back over per-tile digit counts, scatter through
//                    shared memory so that runs of one digit store coalesced
//   k_tree_tiles, k_tree_groups, k_tree_cross   the tree (build_lbvh, minimum_lbvh.h:284-361;
//                    tree.cuh)
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "capi_internal.h"
#include "chain.cuh"
#include "../../include/mlbvh_device.cuh"
#include "climb.cuh"
#include "onesweep.cuh"
#include "sort_leaves.cuh"
#include "tree.cuh"

namespace mlbvh {

namespace {

constexpr int kBoundsThreads = 256;
constexpr int kBoundsMaxBlocks = 1024;
constexpr int kKeysThreads = 256;
// Arrays whose tiles of 1024 keys are all resident at once (3 CTAs on each of
// 148 multiprocessors) sort in those instead of tiles of 4096: a tile's time
// is the chain of its rank steps, and more tiles share the work. Whole builds
// with 1024 / 4096 keys a tile: 16,000 triangles 59 / 73 us, 65,000 72 / 85,
// 213,000 93 / 100, 450,000 124 / 127; beyond, the second wave costs more. The
// small tiles look back 4 at a time (213,000: 1 at a time 100 us, 8 93, 16 93;
// 450,000: 136, 126, 129).
constexpr uint32_t kFewMax = 3 * 148 * sort::kThreads * sort::kFewItems;
constexpr uint32_t kDefaultSpinLimit = 1u << 22;
constexpr int kHdrTreeFlags = 5;  // header word of tree::Scratch::flags; the record count and the next tile follow

// Arrays up to this size take one CTA from the triangles to the sorted keys
// (k_small_sort) instead of the bounds, key and sort kernels, whose launches and
// look-backs cost more than their work. Whole builds, one CTA / chain: 100
// triangles 21 / 36 us, 1,000 24 / 35, 2,000 29 / 38, 4,000 38 / 40; 6,000 52 /
// 42.
constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallMax = 4 * kSmallThreads;

// Scratch layout of one build (offsets from the caller's dScratch). The
// leading region [header, partials) is zeroed by k_scene_bounds on every build.
struct BuildLayout {
    size_t header;     // u32 error word, u32 tile counters[4], u32 tree flags, tree records, next tile
    size_t histogram;  // 4 x 256 u32
    size_t lookback;   // 4 x tiles x 256 u32
    size_t treeCounts; // tree::count_bytes(n)
    size_t partials;   // kBoundsMaxBlocks x 8 floats
    size_t keysA, keysB, valsA, valsB;
    size_t handoff;  // n u32
    size_t summary;  // tree::summary_bytes(n)
    size_t total;
    uint32_t tiles;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

BuildLayout build_layout(uint32_t n)
{
    BuildLayout L;
    const uint32_t sortTile = sort::kThreads * (n <= kFewMax ? sort::kFewItems : sort::kItems);
    L.tiles = (n + sortTile - 1) / sortTile;
    size_t o = 0;
    L.header = o;
    o += 256;
    L.histogram = o;
    o = align256(o + sizeof(uint32_t) * 4 * 256);
    L.lookback = o;
    o = align256(o + sizeof(uint32_t) * 4 * 256 * (size_t)L.tiles);
    L.treeCounts = o;
    o = align256(o + tree::count_bytes(n));
    L.partials = o;
    o = align256(o + sizeof(float) * 8 * kBoundsMaxBlocks);
    L.keysA = o;
    o = align256(o + sizeof(uint32_t) * (size_t)n);
    L.keysB = o;
    o = align256(o + sizeof(uint32_t) * (size_t)n);
    L.valsA = o;
    o = align256(o + sizeof(uint32_t) * (size_t)n);
    L.valsB = o;
    o = align256(o + sizeof(uint32_t) * (size_t)n);
    L.handoff = o;
    o = align256(o + sizeof(uint32_t) * (size_t)n);
    L.summary = o;
    o = align256(o + tree::summary_bytes(n));
    L.total = o;
    return L;
}


// ------------------------------------------------------------ kernels

// Partial bounds of the vertex soup per CTA. The triangles are read as a flat
// float array in 48-byte groups (three float4 = four vertices, axis pattern
// x y z x | y z x y | z x y z), then the scalar tail. Also zeroes the
// counters, histograms and look-back words the sort passes rely on.
__global__ void __launch_bounds__(kBoundsThreads)
    k_scene_bounds(const float* __restrict__ tris, uint32_t n, float* __restrict__ partials,
                   uint32_t* __restrict__ zeroBegin, size_t zeroWords)
{
    chain_begin();
    const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t nthreads = (size_t)gridDim.x * blockDim.x;
    for (size_t i = tid; i < zeroWords; i += nthreads) zeroBegin[i] = 0u;

    float lo[3] = {kFltMax, kFltMax, kFltMax};
    float hi[3] = {-kFltMax, -kFltMax, -kFltMax};
    const size_t nFloats = (size_t)n * 9;
    const size_t nGroups = nFloats / 12;
    const float4* t4 = reinterpret_cast<const float4*>(tris);
    for (size_t g = tid; g < nGroups; g += nthreads) {
        float4 a = __ldg(t4 + 3 * g), b = __ldg(t4 + 3 * g + 1), c = __ldg(t4 + 3 * g + 2);
        lo[0] = fminf(lo[0], fminf(fminf(a.x, a.w), fminf(b.z, c.y)));
        hi[0] = fmaxf(hi[0], fmaxf(fmaxf(a.x, a.w), fmaxf(b.z, c.y)));
        lo[1] = fminf(lo[1], fminf(fminf(a.y, b.x), fminf(b.w, c.z)));
        hi[1] = fmaxf(hi[1], fmaxf(fmaxf(a.y, b.x), fmaxf(b.w, c.z)));
        lo[2] = fminf(lo[2], fminf(fminf(a.z, b.y), fminf(c.x, c.w)));
        hi[2] = fmaxf(hi[2], fmaxf(fmaxf(a.z, b.y), fmaxf(c.x, c.w)));
    }
    for (size_t j = nGroups * 12 + tid; j < nFloats; j += nthreads) {
        float v = __ldg(tris + j);
        int ax = (int)(j % 3);
        lo[ax] = fminf(lo[ax], v);
        hi[ax] = fmaxf(hi[ax], v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    __shared__ float s_box[kBoundsThreads / 32][6];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int a = 0; a < 3; ++a) {
            s_box[warp][a] = lo[a];
            s_box[warp][3 + a] = hi[a];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = s_box[0][threadIdx.x];
        for (int w = 1; w < kBoundsThreads / 32; ++w)
            v = threadIdx.x < 3 ? fminf(v, s_box[w][threadIdx.x]) : fmaxf(v, s_box[w][threadIdx.x]);
        partials[blockIdx.x * 8 + threadIdx.x] = v;
    }
}

// The Morton key of a triangle (buildMortons, minimum_lbvh.cu:68-92).
__device__ __forceinline__ uint32_t triangle_key(const float* t, uint32_t option, f3 lower, f3 upper,
                                                 uint32_t* __restrict__ treeFlags)
{
    const f3 v0 = mk(t[0], t[1], t[2]), v1 = mk(t[3], t[4], t[5]), v2 = mk(t[6], t[7], t[8]);
    const f3 center = (v0 + v1 + v2) / 3.0f;
    if (isnan(center.x) || isnan(center.y) || isnan(center.z)) atomicOr(treeFlags, tree::kNaN);
    const uint32_t key = morton32(lower, upper, center);
    if (!(option & MLBVH_BUILD_OPTION_USE_NORMAL)) return key;
    const f3 ng = normalize(cross(v1 - v0, v2 - v0));
    return (key & 0xFFFFFFC0u) | (morton32(mk(-1, -1, -1), mk(1, 1, 1), ng) >> 26);
}

// The keys of all triangles plus the four digit histograms of the sort. A
// warp takes 32 triangles at a time through its own shared memory with
// coalesced 16-byte loads, the next 32 already on their way, last triangles
// first: the bounds pass has just read the array forwards, so its end is what
// the L2 still holds.
__global__ void __launch_bounds__(kKeysThreads)
    k_keys(const float* __restrict__ tris, uint32_t n, uint32_t option, const float* partials,
           int nPartials, uint32_t* __restrict__ keys, uint32_t* __restrict__ histogram,
           uint32_t* __restrict__ handoff, mlbvh_aabb* __restrict__ sceneOut, uint32_t* __restrict__ treeFlags)
{
    __shared__ float s_scene[6];
    __shared__ uint32_t s_hist[4][256];
    __shared__ float4 s_tri[kKeysThreads / 32][72];  // 32 triangles of 9 floats per warp
    chain_begin();

    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t chunks = (n + 31) / 32, warps = gridDim.x * (kKeysThreads / 32);
    float4 ahead[3];
    auto load = [&](uint32_t c) {  // words 4 lane, 4 lane + 128 and (lanes 0..7) 4 lane + 256 of chunk c
        const size_t base = (size_t)c * 288, words = (size_t)n * 9;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const size_t w = base + 4 * lane + 128 * k;
            if (k == 2 && lane >= 8) break;
            if (w + 4 <= words) {
                ahead[k] = __ldg(reinterpret_cast<const float4*>(tris + w));
            } else {
                float* x = reinterpret_cast<float*>(&ahead[k]);
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = w + j < words ? __ldg(tris + w + j) : 0.0f;
            }
        }
    };
    uint32_t c = blockIdx.x * (kKeysThreads / 32) + warp;  // counted from the last chunk
    if (c < chunks) load(chunks - 1 - c);

    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) (&s_hist[0][0])[i] = 0u;
    if (warp == 0) {
        float lo[3] = {kFltMax, kFltMax, kFltMax}, hi[3] = {-kFltMax, -kFltMax, -kFltMax};
        for (int p = lane; p < nPartials; p += 32) {
            const float4 a = chain_load(reinterpret_cast<const float4*>(partials + p * 8));
            const float4 b = chain_load(reinterpret_cast<const float4*>(partials + p * 8) + 1);
            const float l[3] = {a.x, a.y, a.z}, h[3] = {a.w, b.x, b.y};
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                lo[x] = fminf(lo[x], l[x]);
                hi[x] = fmaxf(hi[x], h[x]);
            }
        }
        for (int o = 16; o > 0; o >>= 1)
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
                hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
            }
        if (lane == 0)
            for (int a = 0; a < 3; ++a) {
                s_scene[a] = lo[a];
                s_scene[3 + a] = hi[a];
            }
    }
    __syncthreads();
    if (blockIdx.x == 0 && sceneOut && threadIdx.x < 6) {
        float* out = reinterpret_cast<float*>(sceneOut);
        out[threadIdx.x] = s_scene[threadIdx.x];
    }
    const f3 lower = mk(s_scene[0], s_scene[1], s_scene[2]);
    const f3 upper = mk(s_scene[3], s_scene[4], s_scene[5]);

    for (; c < chunks; c += warps) {
        const uint32_t chunk = chunks - 1 - c, i = chunk * 32 + lane;
        __syncwarp();
        s_tri[warp][lane] = ahead[0];
        s_tri[warp][lane + 32] = ahead[1];
        if (lane < 8) s_tri[warp][lane + 64] = ahead[2];
        __syncwarp();
        if (c + warps < chunks) load(chunks - 1 - c - warps);
        if (i < n) {
            const uint32_t key = triangle_key(reinterpret_cast<const float*>(s_tri[warp]) + 9 * lane, option, lower,
                                              upper, treeFlags);
            keys[i] = key;
            handoff[i] = 0xFFFFFFFFu;
#pragma unroll
            for (int d = 0; d < 4; ++d) atomicAdd(&s_hist[d][(key >> (8 * d)) & 255u], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
        uint32_t c = (&s_hist[0][0])[i];
        if (c) atomicAdd(&histogram[i], c);
    }
}

// The chain up to the sorted keys for few triangles, in one CTA: scene bounds
// (k_scene_bounds), keys (triangle_key) and four stable passes of 8 bits in
// shared memory, each a warp multisplit over warps of kPer x 32 consecutive
// keys. The same keys, order and words as the kernels above: fminf and fmaxf
// give the same bounds in any order.
template <int kPer>
struct SmallShared {
    uint32_t count[32][256];   // per warp and digit, then the warps' offsets within the digit
    uint32_t part[4][256];     // the same for the four groups of eight warps
    uint32_t start[256];       // first position of each digit
    uint32_t keys[kSmallThreads * kPer], vals[kSmallThreads * kPer];
    float box[32][6];
    uint32_t scan[8];
};
template <int kPer>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_sort(const float* __restrict__ tris, uint32_t n, uint32_t option, uint32_t* __restrict__ header,
                 uint32_t* __restrict__ keysOut, uint32_t* __restrict__ valsOut, uint32_t* __restrict__ handoff,
                 mlbvh_aabb* __restrict__ sceneOut)
{
    extern __shared__ __align__(16) unsigned char smem[];
    SmallShared<kPer>& sh = *reinterpret_cast<SmallShared<kPer>*>(smem);
    chain_begin();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 8) header[tid] = 0u;
    // ---- bounds, as k_scene_bounds
    float lo[3] = {kFltMax, kFltMax, kFltMax}, hi[3] = {-kFltMax, -kFltMax, -kFltMax};
    const uint32_t nFloats = n * 9, nGroups = nFloats / 12;
    const float4* t4 = reinterpret_cast<const float4*>(tris);
    for (uint32_t g = tid; g < nGroups; g += kSmallThreads) {
        const float4 a = __ldg(t4 + 3 * g), b = __ldg(t4 + 3 * g + 1), c = __ldg(t4 + 3 * g + 2);
        lo[0] = fminf(lo[0], fminf(fminf(a.x, a.w), fminf(b.z, c.y)));
        hi[0] = fmaxf(hi[0], fmaxf(fmaxf(a.x, a.w), fmaxf(b.z, c.y)));
        lo[1] = fminf(lo[1], fminf(fminf(a.y, b.x), fminf(b.w, c.z)));
        hi[1] = fmaxf(hi[1], fmaxf(fmaxf(a.y, b.x), fmaxf(b.w, c.z)));
        lo[2] = fminf(lo[2], fminf(fminf(a.z, b.y), fminf(c.x, c.w)));
        hi[2] = fmaxf(hi[2], fmaxf(fmaxf(a.z, b.y), fmaxf(c.x, c.w)));
    }
    for (uint32_t j = nGroups * 12 + tid; j < nFloats; j += kSmallThreads) {
        const float v = __ldg(tris + j);
        const uint32_t ax = j % 3;
#pragma unroll
        for (uint32_t a = 0; a < 3; ++a)
            if (ax == a) {
                lo[a] = fminf(lo[a], v);
                hi[a] = fmaxf(hi[a], v);
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    if (lane == 0)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            sh.box[warp][a] = lo[a];
            sh.box[warp][3 + a] = hi[a];
        }
    __syncthreads();  // also orders the header's zeros before treeFlags below
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = sh.box[lane][a];
        hi[a] = sh.box[lane][3 + a];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    if (sceneOut && tid == 0) {
        float* out = reinterpret_cast<float*>(sceneOut);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            out[a] = lo[a];
            out[3 + a] = hi[a];
        }
    }
    // ---- keys
    const f3 lower = mk(lo[0], lo[1], lo[2]), upper = mk(hi[0], hi[1], hi[2]);
    uint32_t key[kPer], val[kPer], rank[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t i = warp * (32 * kPer) + k * 32 + lane;
        val[k] = i;
        key[k] = 0xFFFFFFFFu;
        if (i < n) {
            float t[9];
#pragma unroll
            for (int j = 0; j < 9; ++j) t[j] = __ldg(tris + 9 * i + j);
            key[k] = triangle_key(t, option, lower, upper, header + kHdrTreeFlags);
            handoff[i] = 0xFFFFFFFFu;
        }
    }
    // ---- four passes
    for (int shift = 0; shift < 32; shift += 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) sh.count[warp][32 * j + lane] = 0u;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = warp * (32 * kPer) + k * 32 + lane;
            const uint32_t d = (key[k] >> shift) & 255u;
            uint32_t peers = __ballot_sync(0xffffffffu, i < n);
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint32_t bit = (d >> b) & 1u;
                const uint32_t m = __ballot_sync(0xffffffffu, bit);
                peers &= bit ? m : ~m;
            }
            const uint32_t before = sh.count[warp][d];
            rank[k] = before + __popc(peers & ((1u << lane) - 1u));
            __syncwarp();
            if (i < n && lane == __ffs(peers) - 1) sh.count[warp][d] = before + __popc(peers);
            __syncwarp();
        }
        __syncthreads();
        {  // eight warps' counts of one digit per thread
            const uint32_t d = tid & 255u, group = tid >> 8;
            uint32_t c = 0;
#pragma unroll
            for (uint32_t w = 0; w < 8; ++w) {
                const uint32_t x = sh.count[8 * group + w][d];
                sh.count[8 * group + w][d] = c;
                c += x;
            }
            sh.part[group][d] = c;
        }
        __syncthreads();
        uint32_t total = 0, inc = 0;
        if (tid < 256) {  // the digits' starts
            uint32_t c = 0;
#pragma unroll
            for (uint32_t g = 0; g < 4; ++g) {
                const uint32_t x = sh.part[g][tid];
                sh.part[g][tid] = c;
                c += x;
            }
            total = inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if ((int)lane >= o) inc += y;
            }
            if (lane == 31) sh.scan[warp] = inc;
        }
        __syncthreads();
        if (tid < 256) {
            for (uint32_t w = 0; w < warp; ++w) inc += sh.scan[w];
            sh.start[tid] = inc - total;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = warp * (32 * kPer) + k * 32 + lane;
            if (i < n) {
                const uint32_t d = (key[k] >> shift) & 255u;
                const uint32_t pos = sh.start[d] + sh.part[warp >> 3][d] + sh.count[warp][d] + rank[k];
                sh.keys[pos] = key[k];
                sh.vals[pos] = val[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const uint32_t i = warp * (32 * kPer) + k * 32 + lane;
            if (i < n) {
                key[k] = sh.keys[i];
                val[k] = sh.vals[i];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t i = warp * (32 * kPer) + k * 32 + lane;
        if (i < n) {
            keysOut[i] = key[k];
            valsOut[i] = val[k];
        }
    }
}

template <int kPer>
mlbvh_status launch_small_sort(const float* tris, uint32_t n, uint32_t option, uint32_t* header, uint32_t* keys,
                               uint32_t* vals, uint32_t* handoff, mlbvh_aabb* scene, cudaStream_t stream)
{
    constexpr int smem = (int)sizeof(SmallShared<kPer>);
    const cudaError_t e =
        cudaFuncSetAttribute(k_small_sort<kPer>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(MLBVH_ERR_LAUNCH, cudaGetErrorString(e));
    k_small_sort<kPer><<<1, kSmallThreads, smem, stream>>>(tris, n, option, header, keys, vals, handoff, scene);
    MLBVH_CHECK_LAUNCH("k_small_sort");
    return MLBVH_OK;
}

}  // namespace

// Just above kFewMax the larger sort tiles need less: the size does not fall
// there, so that scratch for n triangles serves every smaller build.
size_t build_scratch_bytes(uint32_t n)
{
    return std::max(build_layout(n).total, build_layout(std::min(n, kFewMax)).total);
}

mlbvh_status sort_leaves(const mlbvh_triangle* dTris, uint32_t n, uint32_t option, mlbvh_aabb* dScene,
                         uint32_t* dKeysOut, uint32_t* dIdxOut, void* dScratch, cudaStream_t stream,
                         uint32_t spinLimit, SortedLeaves* out)
{
    const BuildLayout L = build_layout(n);
    if (spinLimit == 0) spinLimit = kDefaultSpinLimit;
    char* s = static_cast<char*>(dScratch);
    uint32_t* header = reinterpret_cast<uint32_t*>(s + L.header);
    float* partials = reinterpret_cast<float*>(s + L.partials);
    uint32_t* hist = reinterpret_cast<uint32_t*>(s + L.histogram);
    uint32_t* lookback = reinterpret_cast<uint32_t*>(s + L.lookback);
    uint32_t* keysA = reinterpret_cast<uint32_t*>(s + L.keysA);
    uint32_t* keysB = reinterpret_cast<uint32_t*>(s + L.keysB);
    uint32_t* valsA = reinterpret_cast<uint32_t*>(s + L.valsA);
    uint32_t* valsB = reinterpret_cast<uint32_t*>(s + L.valsB);
    uint32_t* handoff = reinterpret_cast<uint32_t*>(s + L.handoff);
    uint32_t* keysFinal = dKeysOut ? dKeysOut : keysA;
    uint32_t* valsFinal = dIdxOut ? dIdxOut : valsA;
    const float* tris = reinterpret_cast<const float*>(dTris);

    out->keys = keysFinal;
    out->indices = valsFinal;
    out->error = header;
    out->handoff = handoff;
    // after the last pass its inputs are free
    out->tree = tree::place(n, s + L.summary, reinterpret_cast<uint32_t*>(s + L.treeCounts), header + kHdrTreeFlags,
                               keysB);
    out->spinLimit = spinLimit;
    if (n <= kSmallMax)
        return n <= kSmallThreads ? launch_small_sort<1>(tris, n, option, header, keysFinal, valsFinal, handoff, dScene,
                                                         stream)
               : n <= 2 * kSmallThreads
                   ? launch_small_sort<2>(tris, n, option, header, keysFinal, valsFinal, handoff, dScene, stream)
                   : launch_small_sort<4>(tris, n, option, header, keysFinal, valsFinal, handoff, dScene, stream);

    const int sms = device_sm_count();
    const size_t zeroWords = (L.partials - L.header) / 4;
    // at least four vertex groups per thread, and four warp chunks per warp of k_keys: both kernels end in a
    // reduction over their CTAs
    int boundsBlocks = (int)std::min<size_t>(
        (size_t)kBoundsMaxBlocks, std::max<size_t>(1, ((size_t)n * 9 / 48 + kBoundsThreads - 1) / kBoundsThreads));
    boundsBlocks = std::min(boundsBlocks, 4 * sms);
    k_scene_bounds<<<boundsBlocks, kBoundsThreads, 0, stream>>>(tris, n, partials, header, zeroWords);
    MLBVH_CHECK_LAUNCH("k_scene_bounds");
    const int keysBlocks = (int)std::max<uint32_t>(1, std::min<uint32_t>((n + 4 * kKeysThreads - 1) / (4 * kKeysThreads), 4u * sms));
    launch_chained(k_keys, keysBlocks, kKeysThreads, 0, stream, tris, n, option, partials, boundsBlocks, keysA, hist,
                   handoff, dScene, header + kHdrTreeFlags);
    MLBVH_CHECK_LAUNCH("k_keys");

    uint32_t* kin = keysA;
    uint32_t* vin = valsA;
    const bool few = n <= kFewMax;
    const size_t smem = few ? sort::Shape<8, sort::kFewItems>::kSmemBytes : sort::Shape<8>::kSmemBytes;
    for (int pass = 0; pass < 4; ++pass) {
        uint32_t* kout = (pass == 3) ? keysFinal : (pass % 2 == 0 ? keysB : keysA);
        uint32_t* vout = (pass == 3) ? valsFinal : (pass % 2 == 0 ? valsB : valsA);
        const sort::SingleSegment seg{n, L.tiles, hist + 256 * pass};
        using Seg = sort::SingleSegment;
        auto kernel = few ? (pass == 0 ? sort::k_onesweep<8, true, Seg, sort::kFewItems>
                                       : sort::k_onesweep<8, false, Seg, sort::kFewItems>)
                          : (pass == 0 ? sort::k_onesweep<8, true, Seg> : sort::k_onesweep<8, false, Seg>);
        launch_chained(kernel, L.tiles, sort::kThreads, smem, stream, kin, kout, pass == 0 ? nullptr : vin, vout,
                       8 * pass, seg, lookback + (size_t)pass * L.tiles * 256, header + 1 + pass, header, spinLimit);
        MLBVH_CHECK_LAUNCH("k_onesweep");
        kin = kout;
        vin = vout;
    }
    return MLBVH_OK;
}

mlbvh_status build(const mlbvh_triangle* dTris, uint32_t n, uint32_t option, mlbvh_internal_node* dNodes,
                   mlbvh_node_index* dRoot, mlbvh_aabb* dScene, uint32_t* dKeysOut, uint32_t* dIdxOut,
                   uint8_t* dDeltasOut, void* dScratch, size_t scratchBytes, cudaStream_t stream, uint32_t spinLimit)
{
    if (n == 0 || n >= (1u << 30)) return fail(MLBVH_ERR_INVALID_ARG, "nTriangles must be in [1, 2^30)");
    if (!dTris || !dRoot || !dScratch) return fail(MLBVH_ERR_INVALID_ARG, "null triangles, root or scratch pointer");
    if (n > 1 && !dNodes) return fail(MLBVH_ERR_INVALID_ARG, "null internal-node pointer");
    if (!aligned16(dTris) || !aligned16(dNodes) || !aligned16(dScratch) || !aligned16(dRoot) || !aligned16(dScene) ||
        !aligned16(dKeysOut) || !aligned16(dIdxOut) || !aligned16(dDeltasOut))
        return fail(MLBVH_ERR_INVALID_ARG, "device pointers must be 16-byte aligned");
    if (scratchBytes < build_scratch_bytes(n))
        return fail(MLBVH_ERR_INVALID_ARG, "scratch smaller than mlbvh_build_scratch_bytes(n)");
    SortedLeaves sl;
    mlbvh_status st = sort_leaves(dTris, n, option, dScene, dKeysOut, dIdxOut, dScratch, stream, spinLimit, &sl);
    if (st != MLBVH_OK) return st;
    ProfileEvents ev = take_profile_events();
    if (ev.start) cudaEventRecord(ev.start, stream);
    st = tree::launch(reinterpret_cast<const float*>(dTris), tree::OneTree{n}, sl.keys, sl.indices, dNodes, dRoot,
                      dDeltasOut, sl.handoff, sl.tree, device_sm_count(), stream);
    if (st != MLBVH_OK) return st;
    if (ev.stop) cudaEventRecord(ev.stop, stream);
    return MLBVH_OK;
}

mlbvh_status scratch_status(const void* dScratch, cudaStream_t stream)
{
    if (!dScratch) return fail(MLBVH_ERR_INVALID_ARG, "null scratch pointer");
    uint32_t word = 0;
    cudaError_t e = cudaMemcpyAsync(&word, dScratch, sizeof(word), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return fail(MLBVH_ERR_CUDA, cudaGetErrorString(e));
    if (word & 2u)
        return fail(MLBVH_ERR_INVALID_ARG, "batch triangle offsets are not 0 = o[0] < o[1] < ... < o[nMeshes] = "
                                           "nTriangles; nothing was built");
    if (word) return fail(MLBVH_ERR_TIMEOUT, "a bounded device wait gave up; the output of that call is unusable");
    return MLBVH_OK;
}

}  // namespace mlbvh
