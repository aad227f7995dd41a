// detect.cu — self-intersections of a triangulated PLC surface on the GPU.
//
// Replaces cmg::detect::self_intersections (src/detect/self_intersection.cpp:150-188),
// which tests every pair of fan triangles i < j that share no vertex index with the
// Guigue-Devillers orientation test (O. Devillers, P. Guigue, INRIA RR-4488, 2002),
// every decision a sign of the reference's robust::orient3d (the rounded determinant
// unless exactly zero, then the exact sign; coplanar pairs do not cross). Here:
//   1. broad phase: two triangles that cross share a point, so their bounding boxes
//      overlap; the points are rounded to a grid of 2^30 steps, triangles are binned on
//      a uniform grid of cells by their boxes there, and a pair is examined only in the
//      cell that holds the low corner of the intersection of the two boxes, so each
//      candidate pair is seen exactly once. (Here the answer can differ from the
//      reference's: among triangles with coplanar or touching parts, or flat to the
//      rounding of a determinant, its orientation test also names some pairs whose boxes
//      are apart, which share no point; these are left out.)
//   2. middle phase: pairs whose rounded boxes overlap and that share no vertex are dropped
//      when FP32 certifies that one triangle lies on one side of the other's plane; nothing
//      of it is FP64;
//   3. narrow phase, for the pairs left (few, on full warps): the exact boxes, then the
//      same orientation decisions as the reference (o3d_fast in its order, the exact
//      sign when it is zero);
//   4. the crossing pairs are sorted to the reference's (i, j) order on the host, and
//      their rows (facets, corners) gathered on the device.
// The facets are fanned on the device and the surface's extent reduced there, each
// stage's buffers sized once its sizes are known (nothing is uploaded twice).
// The pair set does not depend on the grid, so the result is deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <vector>

#include "cmg_device.cuh"
#include "cmg_exact.cuh"
#include "cmg_util.h"
#include "engine_kernels.h"

namespace cmg::gpu {

namespace {

// The search's frame: points are put on a grid of 2^30 steps over the surface's largest
// extent, and a point's cell is its step times m / 2^32 (monotone, in integers alone).
struct DetGrid {
    double lo[3];
    double span, fx;  // steps = (x - lo) * fx; 0: (x - lo) / span * 2^30
    unsigned m;
    int n[3];
};

__host__ __device__ __forceinline__ double steps_of(double x, double lo, double span, double fx) {
    return fx > 0.0 ? (x - lo) * fx : (x - lo) / span * 1073741824.0;
}

__device__ __forceinline__ int cell_of(int step, unsigned m, int n) {
    return min(static_cast<int>(__umulhi(static_cast<unsigned>(step), m)), n - 1);
}

__device__ __forceinline__ int osign(const d3& a, const d3& b, const d3& c, const d3& d) {
    const double v = o3d_fast(a, b, c, d, nullptr);
    if (v != 0.0) return v > 0.0 ? 1 : -1;
    return exact::orient3d_sign(a, b, c, d);
}

__device__ bool gd_interval(const d3& p1, const d3& q1, const d3& r1, const d3& p2, const d3& q2,
                            const d3& r2) {
    if (osign(q2, p2, p1, q1) > 0) return false;
    if (osign(r2, p2, r1, p1) > 0) return false;
    return true;
}

// Triangle 2's vertex signs (sp, sq, sr) with respect to triangle 1's plane; p1 alone
// on its side of plane 2 after the caller's rotation.
__device__ bool gd_core(const d3& p1, const d3& q1, const d3& r1, const d3& p2, const d3& q2,
                        const d3& r2, int sp, int sq, int sr) {
    if (sp > 0) {
        if (sq > 0) return gd_interval(p1, r1, q1, r2, p2, q2);
        if (sr > 0) return gd_interval(p1, r1, q1, q2, r2, p2);
        return gd_interval(p1, q1, r1, p2, q2, r2);
    }
    if (sp < 0) {
        if (sq < 0) return gd_interval(p1, q1, r1, r2, p2, q2);
        if (sr < 0) return gd_interval(p1, q1, r1, q2, r2, p2);
        return gd_interval(p1, r1, q1, p2, q2, r2);
    }
    if (sq > 0) {
        if (sr >= 0) return gd_interval(p1, r1, q1, q2, r2, p2);
        return gd_interval(p1, q1, r1, p2, q2, r2);
    }
    if (sq < 0) {
        if (sr > 0) return gd_interval(p1, q1, r1, q2, r2, p2);
        return gd_interval(p1, r1, q1, p2, q2, r2);
    }
    if (sr > 0) return gd_interval(p1, q1, r1, r2, p2, q2);
    if (sr < 0) return gd_interval(p1, r1, q1, r2, p2, q2);
    return false;  // coplanar
}

__device__ bool tri_tri_cross(const d3& p1, const d3& q1, const d3& r1, const d3& p2, const d3& q2,
                              const d3& r2) {
    const int a = osign(p1, p2, q2, r2), b = osign(q1, p2, q2, r2), c = osign(r1, p2, q2, r2);
    if (a * b > 0 && a * c > 0) return false;
    const int d = osign(p2, q1, r1, p1), e = osign(q2, q1, r1, p1), f = osign(r2, q1, r1, p1);
    if (d * e > 0 && d * f > 0) return false;
    if (a > 0) {
        if (b > 0) return gd_core(r1, p1, q1, p2, r2, q2, d, f, e);
        if (c > 0) return gd_core(q1, r1, p1, p2, r2, q2, d, f, e);
        return gd_core(p1, q1, r1, p2, q2, r2, d, e, f);
    }
    if (a < 0) {
        if (b < 0) return gd_core(r1, p1, q1, p2, q2, r2, d, e, f);
        if (c < 0) return gd_core(q1, r1, p1, p2, q2, r2, d, e, f);
        return gd_core(p1, q1, r1, p2, r2, q2, d, f, e);
    }
    if (b < 0) {
        if (c >= 0) return gd_core(q1, r1, p1, p2, r2, q2, d, f, e);
        return gd_core(p1, q1, r1, p2, q2, r2, d, e, f);
    }
    if (b > 0) {
        if (c > 0) return gd_core(p1, q1, r1, p2, r2, q2, d, f, e);
        return gd_core(q1, r1, p1, p2, q2, r2, d, e, f);
    }
    if (c > 0) return gd_core(r1, p1, q1, p2, q2, r2, d, e, f);
    if (c < 0) return gd_core(r1, p1, q1, p2, r2, q2, d, f, e);
    return false;  // coplanar
}

// A valid triangle's box in steps (lo.w: 1, or 0 for a triangle to be skipped). The rounding
// is monotone, so triangles whose boxes meet have boxes that meet here.
struct StepBox {
    int4 lo, hi;
};

__global__ void k_det_fixed(int64_t npts, const double* __restrict__ pts, DetGrid G, int4* __restrict__ fpts) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= npts) return;
    int c[3];  // (a point of no valid triangle may be anything)
    for (int q = 0; q < 3; ++q) c[q] = max(__double2int_rn(steps_of(pts[3 * i + q], G.lo[q], G.span, G.fx)), 0);
    fpts[i] = make_int4(c[0], c[1], c[2], 0);
}

// The triangles' boxes, and their cells counted.
__global__ void k_det_count(int64_t ntris, const int* __restrict__ valid, const int* __restrict__ tris,
                            const int4* __restrict__ fpts, DetGrid G, StepBox* __restrict__ fbox,
                            int* __restrict__ cellcnt) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    if (!valid[t]) {
        fbox[t].lo.w = 0;
        return;
    }
    const int4 a = fpts[tris[3 * t]], b = fpts[tris[3 * t + 1]], c = fpts[tris[3 * t + 2]];
    const int4 lo = make_int4(min(a.x, min(b.x, c.x)), min(a.y, min(b.y, c.y)), min(a.z, min(b.z, c.z)), 1);
    const int4 hi = make_int4(max(a.x, max(b.x, c.x)), max(a.y, max(b.y, c.y)), max(a.z, max(b.z, c.z)), 0);
    fbox[t].lo = lo;
    fbox[t].hi = hi;
    const int x0 = cell_of(lo.x, G.m, G.n[0]), x1 = cell_of(hi.x, G.m, G.n[0]);
    const int y0 = cell_of(lo.y, G.m, G.n[1]), y1 = cell_of(hi.y, G.m, G.n[1]);
    const int z0 = cell_of(lo.z, G.m, G.n[2]), z1 = cell_of(hi.z, G.m, G.n[2]);
    for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y)
            for (int x = x0; x <= x1; ++x) atomicAdd(&cellcnt[(z * G.n[1] + y) * G.n[0] + x], 1);
}

// Cell entries (taking the counts down to zero again): the triangle; the cell (below 2^24)
// with, from bit 28, per axis whether it is the triangle's lowest. Of the cells that two
// triangles share, the one with the low corner of their boxes' intersection is the one
// where, on each axis, one of the two has its lowest (cell_of is monotone).
__global__ void k_det_fill(int64_t ntris, const StepBox* __restrict__ fbox, DetGrid G,
                           int* __restrict__ cellcnt, const int64_t* __restrict__ celloff,
                           int2* __restrict__ list) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    const int4 lo = fbox[t].lo, hi = fbox[t].hi;
    if (lo.w == 0) return;
    const int x0 = cell_of(lo.x, G.m, G.n[0]), x1 = cell_of(hi.x, G.m, G.n[0]);
    const int y0 = cell_of(lo.y, G.m, G.n[1]), y1 = cell_of(hi.y, G.m, G.n[1]);
    const int z0 = cell_of(lo.z, G.m, G.n[2]), z1 = cell_of(hi.z, G.m, G.n[2]);
    for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y)
            for (int x = x0; x <= x1; ++x) {
                const int cell = (z * G.n[1] + y) * G.n[0] + x;
                const int low = (x == x0) | (y == y0) << 1 | (z == z0) << 2;
                list[celloff[cell] + atomicSub(&cellcnt[cell], 1) - 1] =
                    make_int2(static_cast<int>(t), cell | low << 28);
            }
}

struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 fixed_diff(const int4& a, const int4& b) {
    return {static_cast<float>(a.x - b.x), static_cast<float>(a.y - b.y), static_cast<float>(a.z - b.z)};
}
__device__ __forceinline__ float max_abs(const V3& a) { return fmaxf(fabsf(a.x), fmaxf(fabsf(a.y), fabsf(a.z))); }

// Whether the corners (a, b, c) certainly have one nonzero orientation with respect to the
// plane through (p, q, r): the reference's rounded determinants have that sign too. In
// fixed-point units each difference is off by at most 1 (two roundings of 1/2, a little
// more with the FP64 product's) and then by u = 2^-24 of itself, d = 1.001 + uD in all with D
// the largest. A 3x3 matrix M that changes of up to d in its entries make singular has
// |det M| <= 12 d D^2, all orders included: with v the singular one's null vector, its largest
// entry 1, M v has entries of at most 3d and can stand in M for that entry's column, and 4 is
// the largest determinant of entries within 1. The FP32 evaluation adds 30 u D^3, the
// reference's rounded determinants 5e-15 D^3 (while none of their products leaves FP64's
// normal range: DetGrid::fx > 0).
__device__ __forceinline__ bool one_side(const int4& p, const int4& q, const int4& r, const int4& a,
                                         const int4& b, const int4& c) {
    const V3 e = fixed_diff(q, p), f = fixed_diff(r, p);
    const V3 wa = fixed_diff(a, p), wb = fixed_diff(b, p), wc = fixed_diff(c, p);
    const float D = fmaxf(fmaxf(max_abs(e), max_abs(f)), fmaxf(max_abs(wa), fmaxf(max_abs(wb), max_abs(wc))));
    const V3 n{e.y * f.z - e.z * f.y, e.z * f.x - e.x * f.z, e.x * f.y - e.y * f.x};
    const float sa = n.x * wa.x + n.y * wa.y + n.z * wa.z;
    const float sb = n.x * wb.x + n.y * wb.y + n.z * wb.z;
    const float sc = n.x * wc.x + n.y * wc.y + n.z * wc.z;
    const float E = D * D * (20.0f + 3.3e-6f * D);
    return fminf(sa, fminf(sb, sc)) > E || fmaxf(sa, fmaxf(sb, sc)) < -E;
}

constexpr int kPairThreads = 128;

// Pairs left by the middle phase that are listed at once (8 GB); a search that leaves more
// takes the cell entries in parts.
constexpr unsigned long long kOpenMost = 1ull << 30;

// One thread per cell entry of [first, last), x of the n in its cell: the pairs with the
// entries x + 1 .. x + n / 2, round the cell's end (each pair once, and the lanes of a cell run
// equally long). Pairs whose boxes meet wait in the warp's list until a full warp examines
// them; what FP32 leaves goes to `open`, nopen of them (more than cap are counted but not
// stored).
//
// One thread per entry testing boxes, cells and orientations in FP64 took 3.02 ms for 512k
// facets (the FP64 pipe 78 % busy, 13 lanes in use): now 80 us, and 40 us for the pairs left.
__global__ void __launch_bounds__(kPairThreads)
k_det_pairs(int64_t first, int64_t last, bool certify, const int2* __restrict__ list, const int64_t* __restrict__ celloff,
            const StepBox* __restrict__ fbox, const int* __restrict__ tris, const int4* __restrict__ fpts,
            int2* __restrict__ open, unsigned long long* __restrict__ nopen, unsigned long long cap) {
    __shared__ int2 s_q[kPairThreads / 32][64];
    int2* queue = s_q[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t e = first + static_cast<int64_t>(blockIdx.x) * kPairThreads + threadIdx.x;
    int2 me = make_int2(0, 0);
    int64_t begin = 0, n = 0;
    if (e < last) {
        me = list[e];
        begin = celloff[me.y & 0xffffff];
        n = celloff[(me.y & 0xffffff) + 1] - begin;
    }
    int4 lo = make_int4(0, 0, 0, 0), hi = lo;
    if (n > 1) {
        lo = fbox[me.x].lo;
        hi = fbox[me.x].hi;
    }
    const auto examine = [&](int q) {
        const int2 pr = queue[q];
        const int a = min(pr.x, pr.y), b = max(pr.x, pr.y);
        int U[3], V[3];
        bool left = true;
        for (int x = 0; x < 3; ++x) {
            U[x] = tris[3 * static_cast<int64_t>(a) + x];
            V[x] = tris[3 * static_cast<int64_t>(b) + x];
        }
        for (int x = 0; x < 3; ++x)
            for (int y = 0; y < 3; ++y) left = left && U[x] != V[y];
        if (left && certify) {
            const int4 p1 = fpts[U[0]], q1 = fpts[U[1]], r1 = fpts[U[2]];
            const int4 p2 = fpts[V[0]], q2 = fpts[V[1]], r2 = fpts[V[2]];
            left = !one_side(p2, q2, r2, p1, q1, r1) && !one_side(p1, q1, r1, p2, q2, r2);
        }
        if (left) {
            const unsigned long long k = atomicAdd(nopen, 1ull);
            if (k < cap) open[k] = make_int2(a, b);
        }
    };
    // a cell's x-th entry of n pairs with (n - 1) / 2 others, the first half of an even n
    // with one more
    const int64_t x = e - begin;
    const int64_t mine = n > 0 ? (n - 1) / 2 + (n % 2 == 0 && x < n / 2) : 0;
    int64_t most = mine;
    for (int o = 16; o > 0; o >>= 1) {
        const int64_t y = __shfl_xor_sync(0xffffffffu, most, o);
        most = y > most ? y : most;
    }
    int held = 0;
    for (int64_t k = 1; k <= most; ++k) {
        bool meet = k <= mine;
        int other = 0;
        if (meet) {
            const int2 f = list[begin + (x + k < n ? x + k : x + k - n)];
            meet = ((me.y | f.y) >> 28 & 7) == 7;
            other = f.x;
        }
        if (meet) {
            const int4 l = fbox[other].lo, h = fbox[other].hi;
            meet = l.x <= hi.x && lo.x <= h.x && l.y <= hi.y && lo.y <= h.y && l.z <= hi.z && lo.z <= h.z;
        }
        const unsigned m = __ballot_sync(0xffffffffu, meet);
        if (meet) queue[held + __popc(m & ((1u << lane) - 1u))] = make_int2(me.x, other);
        held += __popc(m);
        if (held >= 32) {
            __syncwarp();
            held -= 32;
            examine(held + lane);
            __syncwarp();
        }
    }
    __syncwarp();
    if (lane < held) examine(lane);
}

// The pairs left, one per thread: their exact boxes, then the reference's decisions.
__global__ void __launch_bounds__(64)
k_det_cross(const int2* __restrict__ open, const unsigned long long* __restrict__ nopen,
            unsigned long long open_cap, const int* __restrict__ tris, const double* __restrict__ pts, long long* __restrict__ out,
            unsigned long long* __restrict__ nout, unsigned long long cap) {
    const unsigned long long n = *nopen;
    if (n > open_cap) return;  // not all of them are there: the caller runs again
    for (unsigned long long p = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x; p < n;
         p += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        const int a = open[p].x, b = open[p].y;
        const int* U = tris + 3 * static_cast<int64_t>(a);
        const int* V = tris + 3 * static_cast<int64_t>(b);
        auto P = [&](int i) {
            return d3{pts[3 * static_cast<int64_t>(i)], pts[3 * static_cast<int64_t>(i) + 1],
                      pts[3 * static_cast<int64_t>(i) + 2]};
        };
        const d3 p1 = P(U[0]), q1 = P(U[1]), r1 = P(U[2]), p2 = P(V[0]), q2 = P(V[1]), r2 = P(V[2]);
        const auto meet = [](double a1, double b1, double c1, double a2, double b2, double c2) {
            return fmin(a1, fmin(b1, c1)) <= fmax(a2, fmax(b2, c2)) &&
                   fmin(a2, fmin(b2, c2)) <= fmax(a1, fmax(b1, c1));
        };
        if (!meet(p1.x, q1.x, r1.x, p2.x, q2.x, r2.x) || !meet(p1.y, q1.y, r1.y, p2.y, q2.y, r2.y) ||
            !meet(p1.z, q1.z, r1.z, p2.z, q2.z, r2.z))
            continue;
        if (tri_tri_cross(p1, q1, r1, p2, q2, r2)) {
            const unsigned long long k = atomicAdd(nout, 1ull);
            if (k < cap) out[k] = (static_cast<long long>(a) << 32) | static_cast<long long>(b);
        }
    }
}

// ---- fan triangulation of the facets, extent of the surface, result rows ----------

__global__ void k_det_fan_count(const size_t* __restrict__ foff, int64_t nf, int64_t* __restrict__ cnt) {
    const int64_t f = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const int64_t n = static_cast<int64_t>(foff[f + 1] - foff[f]);
    cnt[f] = n >= 3 ? n - 2 : 0;
}

// Fan triangles (v0, v[i-1], v[i]) of facet f at toff[f] + i - 2, with their facet.
__global__ void k_det_fan_emit(const size_t* __restrict__ foff, const int* __restrict__ fidx, int64_t nf,
                               const int64_t* __restrict__ toff, int* __restrict__ tris,
                               int* __restrict__ facet) {
    const int64_t f = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    const size_t o = foff[f];
    const int64_t n = static_cast<int64_t>(foff[f + 1] - o);
    for (int64_t i = 2; i < n; ++i) {
        const int64_t t = toff[f] + i - 2;
        tris[3 * t] = fidx[o];
        tris[3 * t + 1] = fidx[o + i - 1];
        tris[3 * t + 2] = fidx[o + i];
        facet[t] = static_cast<int>(f);
    }
}

// Order-preserving integer image of a double (min / max commute with it).
__device__ __forceinline__ unsigned long long ord_of(double x) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ inline double from_ord(unsigned long long o) {
    const unsigned long long b = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    double d;
    memcpy(&d, &b, sizeof(d));
    return d;
}

struct Extent {
    unsigned long long lo[3], hi[3];  // ord_of images
    double ext_sum;                   // sum of the valid triangles' largest box extents
    unsigned long long nvalid;
    int nonfinite;
};

// Which triangles are valid (indices inside the points), and the surface's extent: minima
// and maxima as integers, one set of atomics per block (per warp, with FP64 comparisons
// and a stored box, 95 us for 512k triangles; now 22 us).
constexpr int kExtThreads = 256;
__global__ void __launch_bounds__(kExtThreads) k_det_extent(int64_t ntris, const int* __restrict__ tris,
                                                            const double* __restrict__ pts, int64_t npts,
                                                            int* __restrict__ valid, Extent* __restrict__ ext) {
    using u64 = unsigned long long;
    __shared__ u64 s_lo[kExtThreads / 32][3], s_hi[kExtThreads / 32][3];
    __shared__ double s_es[kExtThreads / 32];
    __shared__ int s_nv[kExtThreads / 32], s_bad[kExtThreads / 32];
    u64 lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0ull, 0ull, 0ull};
    double sum = 0.0;
    int nv = 0, bad = 0;
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * kExtThreads + threadIdx.x; t < ntris;
         t += static_cast<int64_t>(gridDim.x) * kExtThreads) {
        const int i0 = tris[3 * t], i1 = tris[3 * t + 1], i2 = tris[3 * t + 2];
        const bool ok = i0 >= 0 && i0 < npts && i1 >= 0 && i1 < npts && i2 >= 0 && i2 < npts;
        valid[t] = ok ? 1 : 0;
        if (!ok) continue;
        ++nv;
        double es = 0.0;
        for (int q = 0; q < 3; ++q) {
            const double a = pts[3 * static_cast<int64_t>(i0) + q], b = pts[3 * static_cast<int64_t>(i1) + q],
                         d = pts[3 * static_cast<int64_t>(i2) + q];
            for (const double v : {a, b, d}) bad |= (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
            const u64 x = ord_of(a), y = ord_of(b), z = ord_of(d);
            const u64 l = min(x, min(y, z)), h = max(x, max(y, z));
            lo[q] = min(lo[q], l);
            hi[q] = max(hi[q], h);
            es = fmax(es, from_ord(h) - from_ord(l));
        }
        sum += es;
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int q = 0; q < 3; ++q) {
            lo[q] = min(lo[q], __shfl_xor_sync(0xffffffffu, lo[q], o));
            hi[q] = max(hi[q], __shfl_xor_sync(0xffffffffu, hi[q], o));
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    nv = __reduce_add_sync(0xffffffffu, nv);
    bad = __reduce_or_sync(0xffffffffu, bad);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        for (int q = 0; q < 3; ++q) {
            s_lo[w][q] = lo[q];
            s_hi[w][q] = hi[q];
        }
        s_es[w] = sum;
        s_nv[w] = nv;
        s_bad[w] = bad;
    }
    __syncthreads();
    if (threadIdx.x > 0) return;
    for (int k = 1; k < kExtThreads / 32; ++k) {
        for (int q = 0; q < 3; ++q) {
            lo[q] = min(lo[q], s_lo[k][q]);
            hi[q] = max(hi[q], s_hi[k][q]);
        }
        sum += s_es[k];
        nv += s_nv[k];
        bad |= s_bad[k];
    }
    if (nv == 0) return;
    for (int q = 0; q < 3; ++q) {
        atomicMin(&ext->lo[q], lo[q]);
        atomicMax(&ext->hi[q], hi[q]);
    }
    atomicAdd(&ext->ext_sum, sum);
    atomicAdd(&ext->nvalid, static_cast<u64>(nv));
    if (bad) atomicExch(&ext->nonfinite, 1);
}

// Rows of the sorted pairs: facet_a, facet_b, triangle a's corners, triangle b's.
__global__ void k_det_rows(int64_t np, const long long* __restrict__ keys, const int* __restrict__ tris,
                           const int* __restrict__ facet, int* __restrict__ rows) {
    const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const int64_t a = keys[p] >> 32, b = keys[p] & 0xffffffffll;
    int* r = rows + 8 * p;
    r[0] = facet[a];
    r[1] = facet[b];
    for (int k = 0; k < 3; ++k) {
        r[2 + k] = tris[3 * a + k];
        r[5 + k] = tris[3 * b + k];
    }
}

}  // namespace

namespace {
float g_last_ms = 0.f;  // device time of the last call's broad + narrow phase
}

float self_intersections_last_ms() { return g_last_ms; }

// Sizes one arena for a plan (the plan's pointers are taken again after a growth).
template <typename Plan>
void size_arena(Arena& A, Plan&& plan) {
    A.clear_need();
    plan();
    if (A.overflowed()) {
        A.reserve(A.need());
        plan();
    }
}

void self_intersections(const double* h_pts, int64_t npts, const int* h_fidx, int64_t nidx,
                        const size_t* h_foff, int64_t nfacets, std::vector<int>& rows,
                        cudaStream_t st) {
    rows.clear();
    g_last_ms = 0.f;
    if (nfacets <= 0 || npts <= 0) return;
    if (nidx >= (int64_t(1) << 31)) throw std::invalid_argument("self_intersections: too many facet vertices");
    static std::mutex mu;
    // one arena per stage, each sized when its sizes are known, so that no earlier
    // stage's buffers move: inputs, triangles, cells, entries, output, rows
    static Arena A_in, A_tri, A_cell, A_list, A_out, A_rows;
    static cudaEvent_t ev[2] = {nullptr, nullptr};
    std::lock_guard<std::mutex> lk(mu);
    if (!ev[0])
        for (cudaEvent_t& e : ev) CMG_CUDA(cudaEventCreate(&e));
    const int64_t nf = nfacets;
    double* d_pts;
    int* d_fidx;
    size_t* d_foff;
    int64_t *fcnt, *toff, *stmp_f;
    Extent* ext;
    size_arena(A_in, [&]() {
        A_in.reset();
        d_pts = A_in.take<double>(3 * npts);
        d_fidx = A_in.take<int>(std::max<int64_t>(nidx, 1));
        d_foff = A_in.take<size_t>(nf + 1);
        fcnt = A_in.take<int64_t>(nf);
        toff = A_in.take<int64_t>(nf + 1);
        stmp_f = A_in.take<int64_t>(scan_tmp_elems(nf));
        ext = A_in.take<Extent>(1);
    });
    CMG_CUDA(cudaMemcpyAsync(d_pts, h_pts, sizeof(double) * 3 * npts, cudaMemcpyHostToDevice, st));
    if (nidx) CMG_CUDA(cudaMemcpyAsync(d_fidx, h_fidx, sizeof(int) * nidx, cudaMemcpyHostToDevice, st));
    CMG_CUDA(cudaMemcpyAsync(d_foff, h_foff, sizeof(size_t) * (nf + 1), cudaMemcpyHostToDevice, st));
    CMG_CUDA(cudaEventRecord(ev[0], st));
    const unsigned gf = static_cast<unsigned>((nf + 255) / 256);
    k_det_fan_count<<<gf, 256, 0, st>>>(d_foff, nf, fcnt);
    CMG_LAUNCH();
    exclusive_scan(fcnt, toff, nf, stmp_f, st);
    int64_t ntris = 0;
    CMG_CUDA(cudaMemcpyAsync(&ntris, toff + nf, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CMG_CUDA(cudaStreamSynchronize(st));
    if (ntris < 2) return;
    if (ntris >= (int64_t(1) << 31)) throw std::invalid_argument("self_intersections: too many triangles");

    int *tris, *facet, *valid;
    StepBox* fbox;
    int4* fpts;
    size_arena(A_tri, [&]() {
        A_tri.reset();
        tris = A_tri.take<int>(3 * ntris);
        facet = A_tri.take<int>(ntris);
        valid = A_tri.take<int>(ntris);
        fbox = A_tri.take<StepBox>(ntris);
        fpts = A_tri.take<int4>(npts);
    });
    const unsigned gt = static_cast<unsigned>((ntris + 255) / 256);
    k_det_fan_emit<<<gf, 256, 0, st>>>(d_foff, d_fidx, nf, toff, tris, facet);
    CMG_LAUNCH();
    CMG_CUDA(cudaMemsetAsync(ext, 0, sizeof(Extent), st));
    CMG_CUDA(cudaMemsetAsync(ext->lo, 0xff, sizeof(ext->lo), st));
    k_det_extent<<<std::min<unsigned>(gt, 4 * device_sms()), kExtThreads, 0, st>>>(ntris, tris, d_pts, npts,
                                                                                   valid, ext);
    CMG_LAUNCH();
    Extent h{};
    CMG_CUDA(cudaMemcpyAsync(&h, ext, sizeof(Extent), cudaMemcpyDeviceToHost, st));
    CMG_CUDA(cudaStreamSynchronize(st));
    if (h.nvalid < 2) return;
    if (h.nonfinite) throw std::invalid_argument("self_intersections: non-finite coordinate");
    // grid over the valid triangles' points: cell edge ~ twice the mean box extent, which
    // the multiplier m gives to a quarter of a cell over the span
    double lo[3], hi[3];
    for (int q = 0; q < 3; ++q) {
        lo[q] = from_ord(h.lo[q]);
        hi[q] = from_ord(h.hi[q]);
    }
    DetGrid G{};
    for (int q = 0; q < 3; ++q) {
        G.lo[q] = lo[q];
        G.span = std::max(G.span, hi[q] - lo[q]);
    }
    // (outside this range the certificate does not hold and every pair takes the narrow phase)
    G.fx = G.span > 1e-80 && G.span < 1e90 ? 1073741824.0 / G.span : 0.0;
    double cells = G.span > 0.0 ? std::min(G.span / (2.0 * h.ext_sum / static_cast<double>(h.nvalid)), 2048.0) : 1.0;
    if (!(cells >= 1.0)) cells = 1.0;
    for (;;) {
        G.m = static_cast<unsigned>(4.0 * cells);
        int64_t total = 1;
        for (int q = 0; q < 3; ++q) {
            double top = G.span > 0.0 ? steps_of(hi[q], lo[q], G.span, G.fx) : 0.0;
            if (!(top >= 0.0 && top <= 1073741824.0)) top = 0.0;  // (an extent beyond FP64's range)
            G.n[q] = static_cast<int>((static_cast<uint64_t>(top + 0.5) * G.m >> 32) + 1);
            total *= G.n[q];
        }
        if (total <= (int64_t(1) << 24)) break;
        cells /= 1.5;
    }
    const int64_t ncell = static_cast<int64_t>(G.n[0]) * G.n[1] * G.n[2];

    int* cellcnt;
    int64_t *celloff, *stmp;
    size_arena(A_cell, [&]() {
        A_cell.reset();
        cellcnt = A_cell.take<int>(ncell);
        celloff = A_cell.take<int64_t>(ncell + 1);
        stmp = A_cell.take<int64_t>(scan_tmp_elems(ncell + 1));
    });
    k_det_fixed<<<static_cast<unsigned>((npts + 255) / 256), 256, 0, st>>>(npts, d_pts, G, fpts);
    CMG_LAUNCH();
    CMG_CUDA(cudaMemsetAsync(cellcnt, 0, sizeof(int) * ncell, st));
    k_det_count<<<gt, 256, 0, st>>>(ntris, valid, tris, fpts, G, fbox, cellcnt);
    CMG_LAUNCH();
    exclusive_scan(cellcnt, celloff, ncell, stmp, st);
    int64_t nent = 0;
    CMG_CUDA(cudaMemcpyAsync(&nent, celloff + ncell, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    CMG_CUDA(cudaStreamSynchronize(st));
    int2* list;
    size_arena(A_list, [&]() {
        A_list.reset();
        list = A_list.take<int2>(std::max<int64_t>(nent, 1));
    });
    k_det_fill<<<gt, 256, 0, st>>>(ntris, fbox, G, cellcnt, celloff, list);
    CMG_LAUNCH();
    unsigned long long cap = 1 << 16;
    unsigned long long open_cap = std::max<unsigned long long>(1 << 16, static_cast<unsigned long long>(ntris));
    int64_t part = nent;  // cell entries searched at a time
    for (int attempt = 0; attempt < 64; ++attempt) {  // (once more for each list that was too short)
        long long* out;
        int2* open;
        unsigned long long* counts;  // pairs left by the middle phase, crossing pairs
        size_arena(A_out, [&]() {
            A_out.reset();
            out = A_out.take<long long>(cap);
            open = A_out.take<int2>(open_cap);
            counts = A_out.take<unsigned long long>(2);
        });
        CMG_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), st));
        unsigned long long h_counts[2] = {0, 0};
        for (int64_t e0 = 0; e0 < nent && h_counts[0] <= open_cap; e0 += part) {
            const int64_t e1 = std::min(nent, e0 + part);
            if (e0 > 0) CMG_CUDA(cudaMemsetAsync(counts, 0, sizeof(unsigned long long), st));
            k_det_pairs<<<static_cast<unsigned>((e1 - e0 + kPairThreads - 1) / kPairThreads), kPairThreads, 0, st>>>(
                e0, e1, G.fx > 0.0, list, celloff, fbox, tris, fpts, open, counts, open_cap);
            CMG_LAUNCH();
            k_det_cross<<<4 * device_sms(), 64, 0, st>>>(open, counts, open_cap, tris, d_pts, out, counts + 1,
                                                         cap);
            CMG_LAUNCH();
            if (e1 < nent) {
                CMG_CUDA(cudaMemcpyAsync(h_counts, counts, sizeof(h_counts), cudaMemcpyDeviceToHost, st));
                CMG_CUDA(cudaStreamSynchronize(st));
            }
        }
        CMG_CUDA(cudaEventRecord(ev[1], st));
        CMG_CUDA(cudaMemcpyAsync(h_counts, counts, sizeof(h_counts), cudaMemcpyDeviceToHost, st));
        CMG_CUDA(cudaStreamSynchronize(st));
        CMG_CUDA(cudaEventElapsedTime(&g_last_ms, ev[0], ev[1]));
        const unsigned long long found = h_counts[1];
        if (h_counts[0] > open_cap) {
            if (h_counts[0] <= kOpenMost || part <= kPairThreads) {
                open_cap = h_counts[0];
            } else {
                // fewer entries at a time, by the pairs they left, with a half to spare
                open_cap = std::max(open_cap, kOpenMost);
                const double share = 0.5 * static_cast<double>(open_cap) / static_cast<double>(h_counts[0]);
                part = std::max<int64_t>(kPairThreads, static_cast<int64_t>(share * static_cast<double>(part)));
            }
            continue;
        }
        if (found <= cap) {
            if (found == 0) return;
            // the reference's (i, j) order, then the rows gathered on the device
            std::vector<long long> keys(found);
            CMG_CUDA(cudaMemcpy(keys.data(), out, sizeof(long long) * found, cudaMemcpyDeviceToHost));
            std::sort(keys.begin(), keys.end());
            long long* dkeys;
            int* drows;
            size_arena(A_rows, [&]() {
                A_rows.reset();
                dkeys = A_rows.take<long long>(found);
                drows = A_rows.take<int>(8 * found);
            });
            CMG_CUDA(cudaMemcpyAsync(dkeys, keys.data(), sizeof(long long) * found, cudaMemcpyHostToDevice, st));
            k_det_rows<<<static_cast<unsigned>((found + 255) / 256), 256, 0, st>>>(
                static_cast<int64_t>(found), dkeys, tris, facet, drows);
            CMG_LAUNCH();
            rows.resize(8 * found);
            CMG_CUDA(cudaMemcpyAsync(rows.data(), drows, sizeof(int) * 8 * found, cudaMemcpyDeviceToHost, st));
            CMG_CUDA(cudaStreamSynchronize(st));
            return;
        }
        cap = found;  // exact count known: one more pass with room for every pair
    }
    throw std::runtime_error("self_intersections: output sizing failed");
}

}  // namespace cmg::gpu
