// cmg_seg.cuh — locate the mesh of a flattened index in a batch.
#pragma once

#include "cmg_types.h"

namespace cmg::gpu {

// Largest s with (segs[s].*field) <= idx (segments are in ascending order).
template <int64_t MeshSeg::*field>
__device__ __forceinline__ int find_seg(const MeshSeg* __restrict__ segs, int nseg, int64_t idx) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (segs[mid].*field <= idx) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

}  // namespace cmg::gpu
