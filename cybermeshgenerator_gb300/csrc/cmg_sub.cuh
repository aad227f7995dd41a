// cmg_sub.cuh — the 4^3 sub-bricks of a 16^3 candidate brick.
#pragma once

#include "cmg_types.h"

namespace cmg::gpu {

constexpr int kSub = 4;  // sub-brick edge (cells)

struct SubGeo {
    int x0, y0, z0, x1, y1, z1;
    bool empty;
};

// lb: the brick within its mesh (the bricks of a batch number less than 2^26, so that 64
// sub-bricks each fit the 32-bit work ids).
__device__ __forceinline__ SubGeo sub_geo(const MeshSeg& s, int64_t lb, int sub) {
    SubGeo q;
    const unsigned b = static_cast<unsigned>(lb), bnx = static_cast<unsigned>(s.bnx),
                   bny = static_cast<unsigned>(s.bny);
    const int bx = static_cast<int>(b % bnx);
    const int by = static_cast<int>((b / bnx) % bny);
    const int bz = static_cast<int>(b / (bnx * bny));
    const int per = s.brick / kSub;
    const int sx = sub % per, sy = (sub / per) % per, sz = sub / (per * per);
    q.x0 = bx * s.brick + sx * kSub;
    q.y0 = by * s.brick + sy * kSub;
    q.z0 = (bz + s.bzo) * s.brick + sz * kSub;  // bz counts from the slab's first brick
    q.x1 = min(q.x0 + kSub, s.g.nx);
    q.y1 = min(q.y0 + kSub, s.g.ny);
    q.z1 = min(q.z0 + kSub, s.g.nz);
    // the sub-brick keeps the whole grid's geometry; only its cells inside the slab
    // [z0, z1) are evaluated (none: nothing to do)
    q.empty = q.x0 >= s.g.nx || q.y0 >= s.g.ny || q.z0 >= s.g.nz || q.z1 <= s.g.z0 ||
              q.z0 >= s.g.z1;
    return q;
}

// The centre of the cells [x0, x1) of a brick along one axis, from the grid corner (FP32).
__device__ __forceinline__ float span_centre(int x0, int x1, float h) {
    return __fmul_rn(__fmul_rn(0.5f, static_cast<float>(x0 + x1)), h);
}
// What the ends of FP32's range take from a distance: below 1e-38 a square is rounded to
// multiples of 1.4e-45 (its root moves by up to 1.1e-19), and the reciprocal of a squared
// edge below 3e-39 is infinite (a nearest point moves along an edge of up to 6e-20). The
// bounds of the candidate walk and of the warp-per-sub-brick evaluation hold this much besides
// their relative parts, so that meshes of that size keep all their candidates; at 1e-6 and
// above it rounds away.
constexpr float kTinyDist = 2e-19f;
// Position error of FP32 centroids without their lo parts, over a mesh of that scale.
__device__ __forceinline__ float list_tol(float scale) { return fmaf(8.f * 5.9604645e-8f, scale, kTinyDist); }

}  // namespace cmg::gpu
