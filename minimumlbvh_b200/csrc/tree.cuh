// The agglomerative tree from sorted leaves without hand-offs, shared by the
// single-mesh and the batched builds (build_lbvh, minimum_lbvh.h:284-361; the
// same node words bit for bit).
//
// The tree is fixed by the split deltas alone: internal node p (split between
// leaves p and p + 1) covers the leaves [L, U], L = 1 + the nearest j < p with
// delta(j) >= delta(p), U = the nearest k > p with delta(k) > delta(p) (deltas
// outside the tree count as infinite); its parent is L - 1 when delta(L - 1) <
// delta(U), else U. And a node's box is the join of its leaves' boxes in
// order: the climb joins two children as (right < left ? right : left), so on
// equal values (+0 and -0) the leftmost leaf's wins, whatever the shape of the
// tree below. So every node can be made on its own, from range queries over
// the deltas and the leaf boxes, with no walker waiting on another:
//
//   k_tree_tiles   tiles of 256 leaves, a thread per leaf, resident CTAs that
//     copy the next tile's triangles to shared memory while they work on one.
//     The nearest greater deltas come from per-warp bit masks (one per delta
//     value, 34 of them), the boxes from a table of the joins of 1, 2, 4, 8
//     and 16 consecutive leaves of a warp. A node whose range lies in the tile
//     is interior: it is assembled in shared memory and the tile's nodes are
//     stored as whole 16-byte rows. Roots of the tile's maximal subtrees store
//     themselves into their parents' child slots. Every other node of the tile
//     (its range crosses a tile boundary; 3 % of them) gets a record with the
//     joins of the tile's leaves up to and from its split. The tile also
//     leaves its box, its largest delta and, for every delta value, its first
//     and last leaf of at least that delta.
//   k_tree_groups  the boxes and largest deltas of 32 tiles (groups) and of 32
//     groups (supers), one warp per group (builds of more than 32 tiles).
//   k_tree_cross   a thread per recorded node whose range ends in the tiles
//     beside its own; the others (an eighth) go to 8 lanes each, which pass
//     whole tiles, groups and supers on both sides of the node. Its box is a
//     record's suffix, what was passed, and a record's prefix.
//
// The join is associative only without NaN (right < left is false for either
// order of a NaN). k_keys marks builds with a NaN centroid, and a build whose
// records do not fit (runs of equal keys across tiles, meshes of a few triangles)
// is marked too: those trees are climbed leaf by leaf (climb.cuh), by
// k_tree_groups, or by k_tree_cross in builds that have no groups. Whole builds
// with one NaN (without): 1,000 triangles 43 us (23), 213k 113 (79), 4M 683
// (518); 213k in runs of 300 equal keys 499, 1,000 meshes of 1-16 triangles 134.
//
// Measured (B200, kernel times): 4M-triangle soup 225 + 5 + 34 us against 401
// us for the climb with shared-memory hand-offs per tile; 213k-triangle
// heightfield 18 + 2 + 15 against 47 us; 1,000 triangles 6 + 6 against 24 us;
// 256 meshes of 64-65,536 triangles 180 against 264 us. k_tree_tiles executes
// about 1,000 instructions per 32 leaves at half the issue rate and reads 534
// MB (64-byte DRAM granules for 36-byte triangles in random order), so it is
// bound by issue and barriers, at 40 % of the DRAM rate; few CTAs per SM because
// 5 to 7 (without the copies ahead) left the triangle loads no L1: 275 to 389
// us. k_tree_cross is a chain of 5 to 15 dependent L2 loads.
#pragma once

#include <cstdint>

#include "../../include/mlbvh.h"
#include "../../include/mlbvh_device.cuh"
#include "chain.cuh"
#include "climb.cuh"

namespace mlbvh {
namespace tree {

constexpr uint32_t kTile = 256;  // leaves per tile = threads per CTA
constexpr uint32_t kWarps = kTile / 32;
constexpr uint32_t kInf = 33;  // the delta beyond a tree's ends (real ones are 0..32)
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kStride = kTile + 2;  // staged words: 4 kStride = 8 mod 32, so a row's store reads distinct banks
constexpr uint32_t kNaN = 1u, kFull = 2u;  // flag bits: climb this build instead
constexpr uint32_t kSkip = 4u;             // flag bit: build nothing (bad batch offsets)
// Resident CTAs per SM of k_tree_tiles: 3 leave a thread 75-78 registers; at 4
// (64) whole builds took 60.4 us instead of 58.3 at 65k triangles, 86.5 instead
// of 83.3 at 213k, 181 instead of 179 at 1M and the same 530 at 4M.
constexpr int kTileCtas = 3;
constexpr int kCrossThreads = 128;
constexpr uint32_t kCrossNodes = 64;  // records per CTA and round of k_tree_cross
constexpr uint32_t kGroupThreads = 64;
constexpr int kGroupCtas = 32;  // resident CTAs per SM of k_tree_groups: 2,048 threads
constexpr uint32_t kCrossLanes = 8;  // lanes per crossing node

struct Box {
    f3 lo, hi;
};
__device__ __forceinline__ Box join(const Box& left, const Box& right)
{
    return Box{smin3(right.lo, left.lo), smax3(right.hi, left.hi)};
}

// What a crossing node (or the last leaf of a tree inside a tile) leaves for
// k_tree_cross: {prefix lo, position} {prefix hi, delta | mesh << 8}
// {suffix lo, L} {suffix hi, U}; prefix: the tile's leaves up to the split,
// suffix: those after it. An end that lies outside the tile is kOut | k: the
// node's part of the tile is the suffix of the record k before this one (the
// right end is out) or the prefix of the record k after it (the left end is
// out), or the whole tile where k is 0. A tile's records are in leaf order.
constexpr uint32_t kOut = 0x80000000u;
struct __align__(16) Record {
    float4 w[4];
};

// Per tile, group of 32 tiles, super of 32 groups: box as two float4 and the largest delta.
struct Level {
    float4* box;
    uint8_t* max;
};
// Per tile, its records nearest to either end: of the last leaf whose delta is
// >= d (last[d], d = 0..32) and of the first one whose delta is > d (first[d]),
// counted from the tile's first record; kEdge where that leaf is the tile's
// last. Set for values up to the tile's largest.
constexpr uint32_t kEdge = 255;
struct Ends {
    uint32_t record0, pad;
    uint8_t last[36], first[36];
};

struct Scratch {
    uint32_t* flags;      // kNaN | kFull | kSkip; zeroed before the keys are made
    uint32_t* nRecords;   // zeroed with flags
    uint32_t* nextTile;   // of the climb; zeroed with flags
    Ends* ends;           // per tile
    Record* records;
    uint32_t capacity;    // records
    Level level[3];
    uint32_t* counts;     // finished groups per super; zeroed before
    uint32_t n, nTiles;
};

// bytes of w that are >= d, as 4 bits
__device__ __forceinline__ uint32_t bytes_ge(uint32_t w, uint32_t d)
{
    const uint32_t ge = __vcmpgeu4(w, d * 0x01010101u) & 0x01010101u;
    return (ge | ge >> 7 | ge >> 14 | ge >> 21) & 15u;
}

// Sizes of the summary (bytes) and its place in a scratch region.
inline uint32_t up32(uint32_t x) { return (x + 31) / 32; }
inline uint32_t tiles_of(uint32_t n) { return (uint32_t)(((uint64_t)n + kTile - 1) / kTile); }
inline size_t pad256(size_t x) { return (x + 255) & ~size_t(255); }
inline size_t count_bytes(uint32_t n) { return sizeof(uint32_t) * (size_t)up32(up32(tiles_of(n))); }
inline size_t summary_bytes(uint32_t n)
{
    size_t o = pad256(sizeof(Ends) * (size_t)tiles_of(n));
    uint32_t c = tiles_of(n);
    for (int l = 0; l < 3; ++l) {
        o += pad256(32 * (size_t)c) + pad256(32 * (size_t)up32(c));
        c = up32(c);
    }
    return o;
}
inline Scratch place(uint32_t n, char* summary, uint32_t* counts, uint32_t* flags, void* freeKeys)
{
    Scratch s;
    s.flags = flags;
    s.nRecords = flags + 1;
    s.nextTile = flags + 2;
    s.n = n;
    s.nTiles = tiles_of(n);
    s.counts = counts;
    s.records = static_cast<Record*>(freeKeys);
    s.capacity = n / (sizeof(Record) / sizeof(uint32_t));
    s.ends = reinterpret_cast<Ends*>(summary);
    size_t o = pad256(sizeof(Ends) * (size_t)s.nTiles);
    uint32_t c = s.nTiles;
    for (int l = 0; l < 3; ++l) {
        s.level[l].box = reinterpret_cast<float4*>(summary + o);
        o += pad256(32 * (size_t)c);
        s.level[l].max = reinterpret_cast<uint8_t*>(summary + o);
        o += pad256(32 * (size_t)up32(c));
        c = up32(c);
    }
    return s;
}

// The tree that sorted leaf g belongs to: leaves [start, end), tree `mesh`;
// tree m's nodes lie at `nodes + (start - m)` and are numbered from its first leaf.
struct Segment {
    uint32_t start, end, mesh;
};
struct OneTree {
    static constexpr bool kMany = false;
    uint32_t n;
    __device__ __forceinline__ Segment of(uint32_t) const { return Segment{0u, n, 0u}; }
    __device__ __forceinline__ uint32_t start_of(uint32_t) const { return 0u; }
    __device__ __forceinline__ uint32_t end_of(uint32_t) const { return n; }
};

// Stores child `side` of a node: its name and box.
__device__ __forceinline__ void store_child(mlbvh_internal_node* p, int side, uint32_t name, const Box& b)
{
    float* w = reinterpret_cast<float*>(p);
    p->children[side] = name;
    if (side) {  // bytes 32-55
        *reinterpret_cast<float4*>(w + 8) = make_float4(b.lo.x, b.lo.y, b.lo.z, b.hi.x);
        *reinterpret_cast<float2*>(w + 12) = make_float2(b.hi.y, b.hi.z);
    } else {  // bytes 8-31
        *reinterpret_cast<float2*>(w + 2) = make_float2(b.lo.x, b.lo.y);
        *reinterpret_cast<float4*>(w + 4) = make_float4(b.lo.z, b.hi.x, b.hi.y, b.hi.z);
    }
}

// A leaf's box as build_lbvh forms it (climb.cuh's leaf_box).
__device__ __forceinline__ Box box_of(f3 v0, f3 v1, f3 v2)
{
    const f3 big = mk(kFltMax, kFltMax, kFltMax);
    return Box{smin3(smin3(smin3(big, v0), v1), v2), smax3(smax3(smax3(-big, v0), v1), v2)};
}
__device__ __forceinline__ Box shuffle_xor(const Box& b, int o, uint32_t mask)
{
    return Box{mk(__shfl_xor_sync(mask, b.lo.x, o), __shfl_xor_sync(mask, b.lo.y, o), __shfl_xor_sync(mask, b.lo.z, o)),
               mk(__shfl_xor_sync(mask, b.hi.x, o), __shfl_xor_sync(mask, b.hi.y, o), __shfl_xor_sync(mask, b.hi.z, o))};
}
__device__ __forceinline__ Box shuffle_up(const Box& b, int o)
{
    constexpr uint32_t m = 0xffffffffu;
    return Box{mk(__shfl_up_sync(m, b.lo.x, o), __shfl_up_sync(m, b.lo.y, o), __shfl_up_sync(m, b.lo.z, o)),
               mk(__shfl_up_sync(m, b.hi.x, o), __shfl_up_sync(m, b.hi.y, o), __shfl_up_sync(m, b.hi.z, o))};
}
__device__ __forceinline__ Box shuffle_down(const Box& b, int o)
{
    constexpr uint32_t m = 0xffffffffu;
    return Box{mk(__shfl_down_sync(m, b.lo.x, o), __shfl_down_sync(m, b.lo.y, o), __shfl_down_sync(m, b.lo.z, o)),
               mk(__shfl_down_sync(m, b.hi.x, o), __shfl_down_sync(m, b.hi.y, o), __shfl_down_sync(m, b.hi.z, o))};
}
__device__ __forceinline__ Box load_box(const float4* b, uint32_t i)
{
    const float4 lo = chain_load(b + 2 * (size_t)i), hi = chain_load(b + 2 * (size_t)i + 1);
    return Box{mk(lo.x, lo.y, lo.z), mk(hi.x, hi.y, hi.z)};
}
__device__ __forceinline__ void store_box(float4* b, uint32_t i, const Box& v)
{
    b[2 * (size_t)i] = make_float4(v.lo.x, v.lo.y, v.lo.z, 0.0f);
    b[2 * (size_t)i + 1] = make_float4(v.hi.x, v.hi.y, v.hi.z, 0.0f);
}

// A warp reduces the entries [32 block, ...) of `from` into entry `block` of `to`.
__device__ __forceinline__ void reduce_block(const Level& from, const Level& to, uint32_t entries, uint32_t block)
{
    const uint32_t lane = threadIdx.x & 31, size = min(32u, entries - 32 * block);
    bool has = lane < size;
    Box b{mk(0, 0, 0), mk(0, 0, 0)};
    uint32_t m = 0;
    if (has) {
        b = load_box(from.box, 32 * block + lane);
        m = chain_load(from.max + 32 * (size_t)block + lane);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Box x = shuffle_xor(b, o, 0xffffffffu);
        const bool xhas = __shfl_xor_sync(0xffffffffu, has ? 1 : 0, o) != 0;
        if (!has)
            b = x;
        else if (xhas)
            b = (lane & o) ? join(x, b) : join(b, x);
        has = has || xhas;
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) {
        store_box(to.box, block, b);
        to.max[block] = (uint8_t)m;
    }
}

// The build as a climb (climb.cuh): a thread per leaf, CTAs of kLeaves threads
// that take the tiles in order, each when its last one is done. (A CTA that
// falls behind with tiles of its own is the second to arrive everywhere and
// climbs ever more: 4M triangles with a NaN took 1,072 us with the tiles dealt
// out in turn and take 683 now; 1M in runs of 1,000 equal keys 2,886 us with the
// next tile taken before the last one's climbs end, 1,646 now.)
inline __host__ __device__ bool grouped(const Scratch& sc) { return sc.nTiles > 32; }
template <uint32_t kLeaves, class Trees>
__device__ __forceinline__ void climb_tiles(const float* __restrict__ tris, const Trees& trees, const uint32_t* keys,
                                            const uint32_t* idx, mlbvh_internal_node* __restrict__ nodes,
                                            mlbvh_node_index* __restrict__ roots, uint8_t* __restrict__ deltasOut,
                                            uint32_t* __restrict__ handoff, const Scratch& sc)
{
    __shared__ TileClimbShared<kLeaves> s_climb;
    __shared__ uint32_t s_t0;
    for (;;) {
        __syncthreads();  // no tile is taken before the last one is done
        if (threadIdx.x == 0) s_t0 = atomicAdd(sc.nextTile, 1u) * kLeaves;
        __syncthreads();
        const uint32_t t0 = s_t0;
        if (t0 >= sc.n) return;
        const uint32_t g = t0 + threadIdx.x;
        Segment seg{sc.n, sc.n, 0u};
        uint32_t tri = 0xFFFFFFFFu;
        f3 lo = mk(0.0f, 0.0f, 0.0f), hi = lo;
        if (g < sc.n) {
            seg = trees.of(g);
            tri = chain_load(idx + g);
            // k_tree_tiles leaves before its deltas where a centroid is NaN
            if (deltasOut && g + 1 < seg.end) deltasOut[g] = (uint8_t)delta_at(keys, g);
            // tri >= the tree's size only after a sort whose bounded wait gave up (error word set)
            if (tri < seg.end - seg.start)
                leaf_box(tris + 9 * (size_t)seg.start, seg.end - seg.start, tri, lo, hi);
        }
        tile_climb_prepare(s_climb, keys, sc.n, t0, seg.start, seg.end);
        if (tri < seg.end - seg.start)
            climb_tile(s_climb, t0 - seg.start, seg.end - seg.start, g - seg.start, tri, lo, hi, keys + seg.start,
                       nodes + (seg.start - seg.mesh), handoff + (seg.start - seg.mesh), roots + seg.mesh);
    }
}

// One warp per group; the last group of a super to finish reduces it. Builds
// that cannot take the range queries are climbed here: with 32 registers twice
// as many leaves are under way as k_tree_cross would hold, and the climb is a
// chain of hand-offs.
template <class Trees>
__global__ void __launch_bounds__(kGroupThreads, kGroupCtas)
    k_tree_groups(const float* __restrict__ tris, Trees trees, const uint32_t* keys, const uint32_t* idx,
                  mlbvh_internal_node* __restrict__ nodes, mlbvh_node_index* __restrict__ roots,
                  uint8_t* __restrict__ deltasOut, uint32_t* __restrict__ handoff, Scratch sc)
{
    chain_begin();
    const uint32_t flags = chain_load(sc.flags);
    if (flags) {
        if (!(flags & kSkip)) climb_tiles<kGroupThreads>(tris, trees, keys, idx, nodes, roots, deltasOut, handoff, sc);
        return;
    }
    const uint32_t groups = (sc.nTiles + 31) / 32, g = (blockIdx.x * kGroupThreads + threadIdx.x) >> 5;
    if (g >= groups) return;
    reduce_block(sc.level[0], sc.level[1], sc.nTiles, g);
    if (groups <= 32) return;
    uint32_t last = 0;
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        last = atomicAdd(sc.counts + (g >> 5), 1u) == min(32u, groups - (g & ~31u)) - 1;
        __threadfence();
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();  // the first lane's fence holds for all
    if (last) reduce_block(sc.level[1], sc.level[2], groups, g >> 5);
}

// The next tile's inputs of one thread: its leaf's triangle (copied to shared
// memory as the 48-byte window load_triangle_v reads) and keys.
struct Ahead {
    uint32_t tri, key0, key1;  // sorted triangle; keys of the leaf and its successor
};
__device__ __forceinline__ void copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

template <class Trees>
__global__ void __launch_bounds__(kTile, kTileCtas)
    k_tree_tiles(const float* __restrict__ tris, Trees trees, const uint32_t* keys,
                 const uint32_t* idx, mlbvh_internal_node* __restrict__ nodes,
                 mlbvh_node_index* __restrict__ roots, uint8_t* __restrict__ deltasOut, Scratch sc)
{
    // the joins of 2^k leaves from each leaf on (to the end of its warp), then the assembled nodes by word
    __shared__ __align__(16) float2 s_join[5][3][kTile];
    static_assert(sizeof(float) * 16 * kStride <= sizeof(s_join), "staged nodes fit the table");
    float* const s_node = reinterpret_cast<float*>(s_join);
    __shared__ float4 s_tri[3 * kTile];          // the triangles' windows; a thread reads and fills its own
    __shared__ uint32_t s_ge[kWarps][kInf + 1];  // per warp and delta value d: the leaves whose delta is >= d
    __shared__ uint32_t s_delta[kTile + 1];      // delta(t0 - 1 + j)
    __shared__ uint32_t s_interior[kWarps];      // interior nodes
    __shared__ uint32_t s_cross[kWarps];         // recorded leaves
    __shared__ uint32_t s_rank[kWarps];          // records of the warps before
    __shared__ uint32_t s_any[kInf + 1];         // per delta value d: the warps that hold a delta >= d
    __shared__ uint8_t s_wide[kTile];            // the nodes whose range leaves their warp
    __shared__ uint32_t s_nWide, s_record0;
    __shared__ Box s_warpBox[kWarps], s_before[kWarps], s_after[kWarps];
    __shared__ uint32_t s_mesh[Trees::kMany ? kTile : 1];
    chain_begin();
    if (chain_load(sc.flags) & (kNaN | kSkip)) return;  // the whole CTA: set before this launch

    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = sc.n;
    float4* const window = s_tri + 3 * tid;
    Segment seg{n, n, 0u}, segNext = seg;
    // a triangle's window lies inside its tree's triangles unless it is the last one
    auto windowed = [&](const Segment& s, uint32_t tri) { return s.start + tri + 1 < s.end; };
    auto first_word = [&](const Segment& s, uint32_t tri) { return 9 * ((size_t)s.start + tri); };
    auto load_ahead = [&](uint32_t g, Ahead& a) {
        if (g < n) {
            a.tri = chain_load(idx + g);
            a.key0 = chain_load(keys + g);
            a.key1 = g + 1 < n ? chain_load(keys + g + 1) : 0u;
        }
    };
    auto copy_window = [&](uint32_t g, const Segment& s, Ahead& a) {
        if (g >= n) return;
        if (a.tri >= s.end - s.start) a.tri = 0;  // only after a bounded wait of the sort gave up (error word set)
        if (!windowed(s, a.tri)) return;
        const float* src = tris + (first_word(s, a.tri) & ~(size_t)3);
#pragma unroll
        for (int k = 0; k < 3; ++k) copy16(window + k, src + 4 * k);
    };
    Ahead now{0, 0, 0}, next{0, 0, 0};
    {
        const uint32_t g = blockIdx.x * kTile + tid;
        load_ahead(g, now);
        if (g < n) seg = trees.of(g);
        copy_window(g, seg, now);
        load_ahead(g + gridDim.x * kTile, next);
    }
    if (tid <= kInf) s_any[tid] = 0;
    if (tid == 0) s_nWide = 0;
    __syncthreads();
    for (uint32_t tile = blockIdx.x; tile < sc.nTiles; tile += gridDim.x) {
        const uint32_t t0 = tile * kTile, g = t0 + tid, gNext = g + gridDim.x * kTile;
        const uint32_t last = min(kTile, n - t0) - 1;  // the tile's last leaf
        const bool valid = g < n;
        uint32_t delta = kInf;
        if (valid && g + 1 < seg.end) {
            delta = split_delta(now.key0, now.key1);
            if (deltasOut) deltasOut[g] = (uint8_t)delta;
        }
        s_delta[tid + 1] = delta;
        if (tid == 0) s_delta[0] = t0 > seg.start ? delta_at(keys, t0 - 1) : kInf;
        // masks: lane d makes the one of value d by comparing d with the deltas' bits, 32 leaves at once
        uint32_t equal = 0xffffffffu, ge = 0u;
#pragma unroll
        for (int k = 5; k >= 0; --k) {
            const uint32_t bits = __ballot_sync(0xffffffffu, (delta >> k) & 1u);
            const uint32_t mine = k < 5 ? (uint32_t)((int)(lane << (31 - k)) >> 31) : 0u;  // all ones where d has bit k
            ge |= equal & bits & ~mine;
            equal &= ~(bits ^ mine);
        }
        ge |= equal;
        s_ge[warp][lane] = ge;
        if (ge) atomicOr(&s_any[lane], 1u << warp);
        const uint32_t ge32 = __ballot_sync(0xffffffffu, delta >= 32), ge33 = __ballot_sync(0xffffffffu, delta >= 33);
        if (lane == 0) {
            s_ge[warp][32] = ge32;
            s_ge[warp][33] = ge33;
            if (ge32) atomicOr(&s_any[32], 1u << warp);
            if (ge33) atomicOr(&s_any[33], 1u << warp);
        }
        __syncwarp();
        // the range of node tid where it lies in its warp; the other nodes go to the tile's list
        uint32_t L = 0, U = 0;
        const bool exists = valid && delta < kInf;
        bool inWarp = false;
        if (exists) {
            const uint32_t ml = s_ge[warp][delta] & ((1u << lane) - 1u);
            const uint32_t mr = s_ge[warp][delta + 1] & (0xFFFFFFFEu << lane);
            inWarp = ml != 0u && mr != 0u;
            L = (32 * warp + 32) - (uint32_t)__clz(ml);
            U = 32 * warp + (uint32_t)__ffs(mr) - 1;
        }
        const uint32_t inMask = __ballot_sync(0xffffffffu, inWarp);
        const uint32_t wideMask = __ballot_sync(0xffffffffu, exists && !inWarp);
        // a tree that ends inside the tile: its last leaf's record serves the nodes on both sides
        const uint32_t endMask = __ballot_sync(0xffffffffu, valid && !exists && tid != last);
        uint32_t wide0 = 0;
        if (lane == 0) {
            s_interior[warp] = inMask;
            s_cross[warp] = endMask;
            if (wideMask | endMask) wide0 = atomicAdd(&s_nWide, (uint32_t)__popc(wideMask | endMask));
        }
        wide0 = __shfl_sync(0xffffffffu, wide0, 0);
        if (((wideMask | endMask) >> lane) & 1u)
            s_wide[wide0 + __popc((wideMask | endMask) & ((1u << lane) - 1u))] = (uint8_t)tid;
        if constexpr (Trees::kMany) s_mesh[tid] = seg.mesh;

        // this tile's triangles have arrived; the next one's set out
        Box leaf{mk(kFltMax, kFltMax, kFltMax), mk(-kFltMax, -kFltMax, -kFltMax)};  // no leaf: joins leave it out
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (valid) {
            f3 v0, v1, v2;
            if (windowed(seg, now.tri)) {
                const float4 q0 = window[0], q1 = window[1], q2 = window[2];
                const float f[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
                const uint32_t off = (seg.start + now.tri) & 3u;  // 9 x, modulo 4
                float c[9];
#pragma unroll
                for (int j = 0; j < 9; ++j) {  // two selects by the offset's bits
                    const float x = (off & 1) ? f[j + 1] : f[j], y = (off & 1) ? f[j + 3] : f[j + 2];
                    c[j] = (off & 2) ? y : x;
                }
                v0 = mk(c[0], c[1], c[2]);
                v1 = mk(c[3], c[4], c[5]);
                v2 = mk(c[6], c[7], c[8]);
            } else {
                const float* t = tris + first_word(seg, now.tri);
                v0 = mk(__ldg(t + 0), __ldg(t + 1), __ldg(t + 2));
                v1 = mk(__ldg(t + 3), __ldg(t + 4), __ldg(t + 5));
                v2 = mk(__ldg(t + 6), __ldg(t + 7), __ldg(t + 8));
            }
            leaf = box_of(v0, v1, v2);
        }
        if (gNext < n) segNext = trees.of(gNext);
        copy_window(gNext, segNext, next);

        // the joins of 1, 2, 4, 8, 16 leaves from this one on
        Box run = leaf;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            s_join[k][0][tid] = make_float2(run.lo.x, run.lo.y);
            s_join[k][1][tid] = make_float2(run.lo.z, run.hi.x);
            s_join[k][2][tid] = make_float2(run.hi.y, run.hi.z);
            __syncwarp();
            if (k < 4 && lane + (1u << k) < 32) {
                const uint32_t r = tid + (1u << k);
                const float2 a = s_join[k][0][r], b = s_join[k][1][r], c = s_join[k][2][r];
                run = join(run, Box{mk(a.x, a.y, b.x), mk(b.y, c.x, c.y)});
            }
        }
        auto entry = [&](uint32_t k, uint32_t i) {
            const float2 a = s_join[k][0][i], b = s_join[k][1][i], c = s_join[k][2][i];
            return Box{mk(a.x, a.y, b.x), mk(b.y, c.x, c.y)};
        };
        auto in_warp = [&](uint32_t a, uint32_t b) {  // leaves a..b of one warp: two overlapping runs
            const uint32_t k = min(31u - (uint32_t)__clz(b - a + 1), 4u);
            return join(entry(k, a), entry(k, b + 1 - (1u << k)));
        };
        if (lane == 0) s_warpBox[warp] = join(run, entry(4, tid + 16));
        __syncthreads();

        Box box = leaf;
        if (inWarp) box = in_warp(L, U);
        // the listed nodes, one per thread: node w, range [WL, WU]
        const bool wide = tid < s_nWide;
        uint32_t w = 0, dw = kInf, WL = kNone, WU = kNone;
        Box wbox = leaf, wsuf = leaf;
        if (wide) {
            w = s_wide[tid];
            dw = s_delta[w + 1];
            if (dw < kInf) {
                const uint32_t at = w >> 5;
                uint32_t m = s_ge[at][dw] & ((1u << (w & 31)) - 1u), k = at;
                uint32_t c = s_any[dw] & ((1u << at) - 1u);
                if (m == 0u && c) {
                    k = 31u - (uint32_t)__clz(c);
                    m = s_ge[k][dw];
                }
                if (m)
                    WL = 32 * k + 32 - (uint32_t)__clz(m);
                else if (s_delta[0] >= dw)
                    WL = 0;
                m = s_ge[at][dw + 1] & (0xFFFFFFFEu << (w & 31));
                k = at;
                c = s_any[dw + 1] & (0xFFFFFFFEu << at);
                if (m == 0u && c) {
                    k = (uint32_t)__ffs(c) - 1;
                    m = s_ge[k][dw + 1];
                }
                if (m) WU = 32 * k + (uint32_t)__ffs(m) - 1;
                if (WU > last) WU = kNone;  // none, or past the tree's last leaf (cannot be)
                if (WL != kNone && WU != kNone) {
                    atomicOr(&s_interior[at], 1u << (w & 31));
                    const bool one = (WL >> 5) == (WU >> 5);  // a tree's first or last nodes
                    wbox = in_warp(WL, one ? WU : WL | 31u);
                    for (uint32_t i = (WL >> 5) + 1; i < (WU >> 5); ++i) wbox = join(wbox, s_warpBox[i]);
                    if (!one) wbox = join(wbox, in_warp(WU & ~31u, WU));
                } else {
                    atomicOr(&s_cross[at], 1u << (w & 31));
                }
            }
        }
        const bool recorded = wide && (dw >= kInf || WL == kNone || WU == kNone);
        if (warp == kWarps - 1) {  // the joins of the warps up to and from each warp
            Box p = s_warpBox[min(lane, kWarps - 1)], s = p;
#pragma unroll
            for (int o = 1; o < (int)kWarps; o <<= 1) {
                const Box x = shuffle_up(p, o), y = shuffle_down(s, o);
                if ((int)lane >= o) p = join(x, p);
                if (lane + o < kWarps) s = join(s, y);
            }
            if (lane < kWarps) {
                s_before[lane] = p;
                s_after[lane] = s;
            }
            // the tile's largest delta: the largest value that some warp reaches
            uint32_t m = __ballot_sync(0xffffffffu, s_any[lane] != 0u);
            m = s_any[33] ? 33u : s_any[32] ? 32u : 31u - (uint32_t)__clz(m);
            if (lane == 0) {  // the tile's summary
                store_box(sc.level[0].box, tile, s);
                sc.level[0].max[tile] = (uint8_t)m;
            }
        }
        // the tile's ends: two warps, lane d for value d (last[0] is always the tile's last leaf)
        uint32_t tileEnd = last;
        if (warp == kWarps - 2) {
            const uint32_t c = s_any[lane + 1];
            if (c) {
                const uint32_t k = 31u - (uint32_t)__clz(c);
                tileEnd = 32 * k + 31 - (uint32_t)__clz(s_ge[k][lane + 1]);
            }
        } else if (warp == kWarps - 3) {
            const uint32_t c = s_any[lane + 1];
            if (c) {
                const uint32_t k = (uint32_t)__ffs(c) - 1;
                tileEnd = 32 * k + (uint32_t)__ffs(s_ge[k][lane + 1]) - 1;
            }
        } else if (tid == kTile - 128 && s_any[33]) {  // first[32]
            const uint32_t k = (uint32_t)__ffs(s_any[33]) - 1;
            tileEnd = 32 * k + (uint32_t)__ffs(s_ge[k][33]) - 1;
        }
        __syncthreads();
        if (recorded) {  // the joins of the tile's leaves up to the split and after it
            const uint32_t at = w >> 5;
            wbox = in_warp(32 * at, w);
            if (at > 0) wbox = join(s_before[at - 1], wbox);
            if (w < last) {
                if ((w & 31) < 31) {
                    wsuf = in_warp(w + 1, w | 31u);
                    if (at + 1 < kWarps) wsuf = join(wsuf, s_after[at + 1]);
                } else {
                    wsuf = s_after[at + 1];
                }
            }
        }
        if (warp == kWarps - 1) {  // the tile's records get their place
            const uint32_t c = lane < kWarps ? (uint32_t)__popc(s_cross[lane]) : 0u;
            uint32_t up = c;
#pragma unroll
            for (int o = 1; o < (int)kWarps; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, up, o);
                if ((int)lane >= o) up += x;
            }
            if (lane < kWarps) s_rank[lane] = up - c;
            if (lane == kWarps - 1) {
                const uint32_t r = up ? atomicAdd(sc.nRecords, up) : 0u;
                if (r + up > sc.capacity) atomicOr(sc.flags, kFull);
                s_record0 = r;
                sc.ends[tile].record0 = r;
                sc.ends[tile].last[0] = kEdge;
            }
        }
        // the record of leaf `i` of the tile, from the tile's first
        auto rank_of = [&](uint32_t i) {
            return s_rank[i >> 5] + (uint32_t)__popc(s_cross[i >> 5] & ((1u << (i & 31)) - 1u));
        };
        __syncthreads();  // the table is read; its space takes the nodes

        if (recorded) {
            const uint32_t rank = rank_of(w), slot = s_record0 + rank;
            uint32_t l = kOut, u = kOut;
            if (WL != kNone) {
                l = t0 + WL;
                if (WL > 0) u = kOut | (rank - rank_of(WL - 1));
            } else if (WU != kNone) {
                u = t0 + WU;
                if (WU < last) l = kOut | (rank_of(WU) - rank);
            }
            const uint32_t mesh = Trees::kMany ? s_mesh[Trees::kMany ? w : 0] : 0u;
            if (slot < sc.capacity) {
                float4* r = sc.records[slot].w;
                r[0] = make_float4(wbox.lo.x, wbox.lo.y, wbox.lo.z, __uint_as_float(t0 + w));
                r[1] = make_float4(wbox.hi.x, wbox.hi.y, wbox.hi.z, __uint_as_float(dw | mesh << 8));
                r[2] = make_float4(wsuf.lo.x, wsuf.lo.y, wsuf.lo.z, __uint_as_float(l));
                r[3] = make_float4(wsuf.hi.x, wsuf.hi.y, wsuf.hi.z, __uint_as_float(u));
            }
        }
        // each subtree's root stores itself into its parent (returned, with the tile's first leaf as 0): in shared
        // memory, except where the parent lies in the tile before
        auto place = [&](uint32_t lo, uint32_t hi, uint32_t mesh, uint32_t child, const Box& b) -> uint32_t {
            const uint32_t dl = s_delta[lo], dr = s_delta[hi + 1];
            const int side = dl < dr ? 1 : 0;
            const uint32_t q = side ? lo - 1 : hi;
            if (dl >= kInf && dr >= kInf) {  // the whole tree
                roots[mesh] = child;
                return kNone - 1;
            }
            if (q == kNone) {
                store_child(nodes + (t0 - 1 - mesh), side, child, b);
                return q;
            }
            float* x = s_node + q;
            x[side * kStride] = __uint_as_float(child);
            x += (2 + 6 * side) * kStride;
            x[0 * kStride] = b.lo.x;
            x[1 * kStride] = b.lo.y;
            x[2 * kStride] = b.lo.z;
            x[3 * kStride] = b.hi.x;
            x[4 * kStride] = b.hi.y;
            x[5 * kStride] = b.hi.z;
            return q;
        };
        auto place_node = [&](uint32_t i, uint32_t lo, uint32_t hi, const Segment& sg, const Box& b) {
            const uint32_t q = place(lo, hi, sg.mesh, t0 + i - sg.start, b);
            const uint32_t end = t0 + hi - sg.start, inner = sg.end - sg.start - 1;
            s_node[14 * kStride + i] = __uint_as_float(q == kNone - 1 ? kInvalid : t0 + q - sg.start);
            s_node[15 * kStride + i] = __uint_as_float(end < inner ? end : 0xFFFFFFFFu);
        };
        if (valid) place(tid, tid, seg.mesh, kLeafBit | now.tri, leaf);
        if (inWarp) place_node(tid, L, U, seg, box);
        if (wide && !recorded) {
            Segment sg = seg;
            if constexpr (Trees::kMany) sg = Segment{trees.start_of(s_mesh[w]), trees.end_of(s_mesh[w]), s_mesh[w]};
            place_node(w, WL, WU, sg, wbox);
        }
        {
            Ends* e = sc.ends + tile;
            const uint8_t r = tileEnd < last ? (uint8_t)rank_of(tileEnd) : (uint8_t)kEdge;
            if (warp == kWarps - 2)
                e->last[lane + 1] = r;
            else if (warp == kWarps - 3)
                e->first[lane] = r;
            else if (tid == kTile - 128)
                e->first[32] = r;
        }
        if (tid <= kInf) s_any[tid] = 0;
        if (tid == 0) s_nWide = 0;
        __syncthreads();
        // a crossing node's child that lies in the tile
        if (recorded && dw < kInf && (WL != kNone || WU != kNone)) {
            const int side = WL != kNone ? 0 : 1;
            const float* x = s_node + w;
            const float* y = x + (2 + 6 * side) * kStride;
            store_child(nodes + (t0 + w - (Trees::kMany ? s_mesh[Trees::kMany ? w : 0] : 0u)), side,
                        __float_as_uint(x[side * kStride]),
                        Box{mk(y[0], y[kStride], y[2 * kStride]), mk(y[3 * kStride], y[4 * kStride], y[5 * kStride])});
        }
        // the interior nodes, 16 bytes per thread and step
        float4* const out = reinterpret_cast<float4*>(nodes);
#pragma unroll
        for (uint32_t c = 0; c < 4; ++c) {
            const uint32_t i = c * (kTile / 4) + (tid >> 2), row = tid & 3;
            if ((s_interior[i >> 5] >> (i & 31)) & 1u) {
                const float* w = s_node + 4 * row * kStride + i;
                const size_t at = t0 + i - (Trees::kMany ? s_mesh[Trees::kMany ? i : 0] : 0u);
                out[4 * at + row] = make_float4(w[0], w[kStride], w[2 * kStride], w[3 * kStride]);
            }
        }
        seg = segNext;
        now = next;
        load_ahead(gNext + gridDim.x * kTile, next);
        __syncthreads();  // the stored nodes' space takes the next table
    }
}

// ------------------------------------------------------- crossing nodes
// 8 lanes per node: 4 look left of its tile, 4 right (the same instructions;
// `left` tells them apart). r = 0..3 is the lane's place among its 4, `lanes`
// their mask.
struct Side {
    bool left;
    uint32_t r, lanes;
};
__device__ __forceinline__ Level level_of(const Scratch& sc, int l)
{
    return Level{l == 0 ? sc.level[0].box : l == 1 ? sc.level[1].box : sc.level[2].box,
                 l == 0 ? sc.level[0].max : l == 1 ? sc.level[1].max : sc.level[2].max};
}
// The join of what a side has passed, nearest to farthest from the node's tile.
struct Sum {
    Box b;
    bool has;
};
// Joins entries [from, to] of one block of a level (8 per lane, those outside
// replaced by the nearest inside: joining an entry twice changes nothing) onto
// acc's outer end. Every lane of the side gets the result.
__device__ __forceinline__ void join_entries(Sum& acc, const float4* boxes, uint32_t from, uint32_t to,
                                             const Side& sd)
{
    const uint32_t base = (from & ~31u) + 8 * sd.r;
    Box mine;
#pragma unroll
    for (uint32_t h = 0; h < 8; h += 4) {
        Box x[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) x[k] = load_box(boxes, min(max(base + h + k, from), to));
        const Box y = join(join(x[0], x[1]), join(x[2], x[3]));
        mine = h == 0 ? y : join(mine, y);
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        const Box x = shuffle_xor(mine, o, sd.lanes);
        mine = (sd.r & o) ? join(x, mine) : join(mine, x);
    }
    acc.b = !acc.has ? mine : sd.left ? join(mine, acc.b) : join(acc.b, mine);
    acc.has = true;
}

// The nearest tile on the side of tile i whose largest delta is >= d: block by
// block up the levels and down again; the entries passed over are joined onto
// acc. kNone: none (left only: a tree's last leaf has an infinite delta).
__device__ __forceinline__ uint32_t find_tile(const Scratch& sc, uint32_t i, uint32_t d, Sum& acc, const Side& sd)
{
    auto entries = [&](int l) { return (sc.nTiles + (1u << (5 * l)) - 1) >> (5 * l); };
    auto scan = [&](int l, uint32_t base, uint32_t allowed) -> uint32_t {
        allowed &= 0xFFFFFFFFu >> (32u - min(32u, entries(l) - base));
        if (allowed == 0u) return kNone;
        const Level level = level_of(sc, l);
        const uint2 w = chain_load(reinterpret_cast<const uint2*>(level.max + base) + sd.r);
        uint32_t m = (bytes_ge(w.x, d) | bytes_ge(w.y, d) << 4) << (8 * sd.r);
        m |= __shfl_xor_sync(sd.lanes, m, 1);
        m |= __shfl_xor_sync(sd.lanes, m, 2);
        m &= allowed;
        uint32_t found = kNone;
        if (m) {
            const uint32_t bit = sd.left ? 31u - (uint32_t)__clz(m) : (uint32_t)__ffs(m) - 1u;
            found = base + bit;
            allowed &= sd.left ? 0xFFFFFFFEu << bit : (1u << bit) - 1u;
        }
        if (allowed)
            join_entries(acc, level.box, base + (uint32_t)__ffs(allowed) - 1u, base + 31u - (uint32_t)__clz(allowed),
                         sd);
        return found;
    };
    int l = 0;
    uint32_t found;
    for (;; ++l, i >>= 5) {
        uint32_t base = i & ~31u;
        found = scan(l, base, sd.left ? (1u << (i & 31u)) - 1u : 0xFFFFFFFEu << (i & 31u));
        if (found != kNone) break;
        if (l == 2) {  // the top level is walked block by block
            while (found == kNone && (sd.left ? base > 0u : base + 32u < entries(2))) {
                base = sd.left ? base - 32u : base + 32u;
                found = scan(2, base, 0xFFFFFFFFu);
            }
            break;
        }
        if (entries(l) <= 32u) return kNone;
    }
    while (found != kNone && l > 0) {
        --l;
        found = scan(l, 32u * found, 0xFFFFFFFFu);
    }
    return found;
}

template <class Trees>
__global__ void __launch_bounds__(kCrossThreads)
    k_tree_cross(const float* __restrict__ tris, Trees trees, const uint32_t* keys,
                 const uint32_t* idx, mlbvh_internal_node* __restrict__ nodes,
                 mlbvh_node_index* __restrict__ roots, uint8_t* __restrict__ deltasOut, uint32_t* __restrict__ handoff,
                 Scratch sc)
{
    __shared__ uint32_t s_far[kCrossNodes], s_nFar;
    chain_begin();
    const uint32_t flags = chain_load(sc.flags);
    if (flags & kSkip) return;
    if (flags) {  // NaN or too many records: every leaf climbs
        if (!grouped(sc)) climb_tiles<kCrossThreads>(tris, trees, keys, idx, nodes, roots, deltasOut, handoff, sc);
        return;
    }
    const uint32_t count = min(chain_load(sc.nRecords), sc.capacity);
    struct Half {  // a record's half, or a tile's box
        Box b;
        uint32_t x, y;
    };
    auto load_half = [&](const float4* r) {
        const float4 a = chain_load(r), b = chain_load(r + 1);
        return Half{Box{mk(a.x, a.y, a.z), mk(b.x, b.y, b.z)}, __float_as_uint(a.w), __float_as_uint(b.w)};
    };
    auto tile_box = [&](uint32_t t) { return (const float4*)(sc.level[0].box + 2 * (size_t)t); };
    auto prefix_of = [&](uint32_t slot) { return (const float4*)sc.records[slot].w; };
    // the part of a range in the node's own tile
    auto own_part = [&](uint32_t slot, uint32_t tile, uint32_t l, uint32_t u) {
        const uint32_t k = (l & kOut ? l : u) & 0xFFu;
        const bool suffix = !(l & kOut);
        return load_half(k == 0u ? tile_box(tile) : suffix ? prefix_of(slot - k) + 2 : prefix_of(slot + k)).b;
    };
    // A range's end in tile t beyond its own on one side (the tile holds it):
    // where, the delta there, and the tile's part of the range joined onto acc.
    struct End {
        uint32_t at, delta;
    };
    auto end_in = [&](uint32_t t, bool left, uint32_t record0, uint32_t rank, Sum& acc) {
        End e;
        Half x;
        if (rank == kEdge) {  // the split after the tile's last leaf
            const uint32_t at = min((t + 1) * kTile, sc.n) - 1;
            e = End{left ? at + 1 : at, kNone};
            if (left) return e;  // nothing of the tile
            x = load_half(tile_box(t));
        } else {
            const float4* r = prefix_of(record0 + rank);
            x = load_half(r);
            e = End{left ? x.x + 1 : x.x, x.y & 0xFFu};
            if (left) x = load_half(r + 2);
        }
        acc.b = !acc.has ? x.b : left ? join(x.b, acc.b) : join(acc.b, x.b);
        acc.has = true;
        return e;
    };
    auto finish = [&](uint32_t p, uint32_t mesh, End l, End u, const Box& box) {
        const uint32_t start = trees.start_of(mesh), end = trees.end_of(mesh), inner = end - start - 1;
        if (l.delta == kNone) l.delta = l.at > start ? delta_at(keys, l.at - 1) : kInf;
        if (u.delta == kNone) u.delta = u.at + 1 < end ? delta_at(keys, u.at) : kInf;
        uint32_t parent = kInvalid;
        if (l.delta >= kInf && u.delta >= kInf) {
            roots[mesh] = p - start;
        } else {
            const int side = l.delta < u.delta ? 1 : 0;
            const uint32_t at = side ? l.at - 1 : u.at;
            store_child(nodes + (at - mesh), side, p - start, box);
            parent = at - start;
        }
        const uint32_t last = u.at - start;
        *reinterpret_cast<uint2*>(&nodes[p - mesh].parent) = make_uint2(parent, last < inner ? last : 0xFFFFFFFFu);
    };
    for (uint32_t base = blockIdx.x * kCrossNodes; base < count; base += gridDim.x * kCrossNodes) {
        __syncthreads();  // the last round's list is read
        if (threadIdx.x == 0) s_nFar = 0;
        __syncthreads();
        // ranges that end in the tiles beside the node's own; what they may need of those tiles is loaded at once
        const uint32_t slot = base + threadIdx.x;
        if (threadIdx.x < kCrossNodes && slot < count) {
            const Half pre = load_half(prefix_of(slot)), suf = load_half(prefix_of(slot) + 2);
            const uint32_t p = pre.x, d = pre.y & 0xFFu, mesh = pre.y >> 8, l = suf.x, u = suf.y, tile = p / kTile;
            if (d < kInf) {  // else a tree's last leaf, no node
                const uint32_t tl = max(tile, 1u) - 1, tr = min(tile + 1, sc.nTiles - 1);
                const uint32_t maxL = chain_load(sc.level[0].max + tl), maxR = chain_load(sc.level[0].max + tr);
                const uint32_t recL = chain_load(&sc.ends[tl].record0), recR = chain_load(&sc.ends[tr].record0);
                const uint32_t rankL = chain_load(sc.ends[tl].last + d), rankR = chain_load(sc.ends[tr].first + d);
                Sum acc{own_part(slot, tile, l, u), true};
                const bool nearL = !(l & kOut) || tile == 0 || maxL >= d, nearR = !(u & kOut) || maxR > d;
                if (nearL && nearR) {
                    End el{l, kNone}, eu{u, kNone};
                    if (l & kOut) el = tile == 0 ? End{0u, kInf} : end_in(tl, true, recL, rankL, acc);
                    if (u & kOut) eu = end_in(tr, false, recR, rankR, acc);
                    finish(p, mesh, el, eu, acc.b);
                } else {
                    s_far[atomicAdd(&s_nFar, 1u)] = slot;
                }
            }
        }
        __syncthreads();
        // the others: 8 lanes each, 4 to a side
        const uint32_t q = threadIdx.x % kCrossLanes, nFar = s_nFar;
        const Side sd{q < 4, q & 3u, 0xFu << (threadIdx.x & 28u)};
        const uint32_t both = 0xFFu << (threadIdx.x & 24u);
        for (uint32_t i = threadIdx.x / kCrossLanes; i < nFar; i += kCrossThreads / kCrossLanes) {
            const uint32_t far = s_far[i];
            const Half pre = load_half(prefix_of(far)), suf = load_half(prefix_of(far) + 2);
            const uint32_t p = pre.x, d = pre.y & 0xFFu, mesh = pre.y >> 8, l = suf.x, u = suf.y, tile = p / kTile;
            const Box own = own_part(far, tile, l, u);
            // the range's end on this lane's side, and what lies between
            Sum acc{Box{mk(0, 0, 0), mk(0, 0, 0)}, false};
            End e{sd.left ? l : u, kNone};
            if (e.at & kOut) {
                const uint32_t t = find_tile(sc, tile, sd.left ? d : d + 1, acc, sd);
                e = End{sd.left ? 0u : sc.n - 1, kInf};
                if (t != kNone)
                    e = end_in(t, sd.left, chain_load(&sc.ends[t].record0),
                               sd.left ? chain_load(sc.ends[t].last + d) : chain_load(sc.ends[t].first + d), acc);
            }
            const Box other = shuffle_xor(acc.b, 4, both);
            const bool otherHas = __shfl_xor_sync(both, acc.has ? 1 : 0, 4) != 0;
            const End otherEnd{__shfl_xor_sync(both, e.at, 4), __shfl_xor_sync(both, e.delta, 4)};
            if (q == 0) {  // a left lane: acc is the left part, other the right one
                Box box = acc.has ? join(acc.b, own) : own;
                if (otherHas) box = join(box, other);
                finish(p, mesh, e, otherEnd, box);
            }
        }
    }
}

// Launches the kernels after the sort's (chain.cuh). handoff: n words of ~0 (the climb's).
template <class Trees>
inline mlbvh_status launch(const float* tris, const Trees& trees, const uint32_t* keys, const uint32_t* idx,
                           mlbvh_internal_node* nodes, mlbvh_node_index* roots, uint8_t* deltasOut, uint32_t* handoff,
                           const Scratch& sc, int sms, cudaStream_t stream)
{
    const uint32_t tileBlocks = std::min<uint32_t>(sc.nTiles, kTileCtas * (uint32_t)sms);
    launch_chained(k_tree_tiles<Trees>, tileBlocks, kTile, 0, stream, tris, trees, keys, idx, nodes, roots, deltasOut,
                   sc);
    MLBVH_CHECK_LAUNCH("k_tree_tiles");
    uint32_t blocks = std::min<uint32_t>(sc.n / 24 / kCrossNodes + 1, 32u * (uint32_t)sms);
    // a kernel that may have to climb gets a thread per leaf, up to what is resident
    if (grouped(sc)) {
        const uint32_t leafBlocks =
            std::max(std::min<uint32_t>((sc.n + kGroupThreads - 1) / kGroupThreads, kGroupCtas * (uint32_t)sms),
                     (up32(sc.nTiles) + kGroupThreads / 32 - 1) / (kGroupThreads / 32));
        launch_chained(k_tree_groups<Trees>, leafBlocks, kGroupThreads, 0, stream, tris, trees, keys, idx, nodes, roots,
                       deltasOut, handoff, sc);
        MLBVH_CHECK_LAUNCH("k_tree_groups");
    } else {
        blocks = std::max<uint32_t>(blocks, (sc.n + kCrossThreads - 1) / kCrossThreads);
    }
    launch_chained(k_tree_cross<Trees>, blocks, kCrossThreads, 0, stream, tris, trees, keys, idx, nodes, roots,
                   deltasOut, handoff, sc);
    MLBVH_CHECK_LAUNCH("k_tree_cross");
    return MLBVH_OK;
}

}  // namespace tree
}  // namespace mlbvh
