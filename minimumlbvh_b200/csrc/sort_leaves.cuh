// The build chain up to the sorted leaves, shared by the LBVH and PLOC builds.
#pragma once

#include "capi_internal.h"
#include "tree.cuh"

namespace mlbvh {

// The build chain up to the sorted leaves (scene bounds, keys, four stable
// sort passes), shared by build() and build_ploc(); the caller has checked
// the arguments. Pointers into the caller's scratch (or its outputs).
struct SortedLeaves {
    const uint32_t* keys;     // n sorted Morton keys
    const uint32_t* indices;  // n triangle indices in that order
    uint32_t* error;          // the build's error word (scratch offset 0)
    uint32_t* handoff;        // n words of ~0 (the climb's)
    tree::Scratch tree;
    uint32_t spinLimit;       // polls per bounded wait
};
mlbvh_status sort_leaves(const mlbvh_triangle* dTris, uint32_t n, uint32_t option, mlbvh_aabb* dScene,
                         uint32_t* dKeysOut, uint32_t* dIdxOut, void* dScratch, cudaStream_t stream,
                         uint32_t spinLimit, SortedLeaves* out);

}  // namespace mlbvh
