// occupancy.cu — inside/outside bytes by exact vertical ray parity.
//
// Restates the reference's classify_occupancy (src/voxelize/voxelize.cpp:121-196)
// for the GPU:
//   k_tri_prep     triangle soup (80-byte records) + the reference's xy cell box of
//                  each triangle (floor((x-corner)/h), clamped; voxelize.cpp:82-100)
//   k_col_pairs    (triangle, column) pairs of those boxes -> per-column buckets (CSR)
//   k_occ_filter   one CTA per row of 32 columns, lanes over the row's bucket entries:
//                  the segment test in FP32 with a certified error bound; the crossings'
//                  heights and the entries that FP32 leaves (orient3d in reference
//                  operation order, FP64, no FMA) as dense lists; every column whose
//                  evaluations are all decided by the rounded determinant is finished
//                  here (crossings in shared memory, parity, coalesced byte rows);
//                  the rest are appended to a compact list
//   k_occ_exact    one warp per listed column: the same walk with exact signs for the
//                  undecided evaluations, the reference's six nudges on a graze, and
//                  its keep-the-last-partial-result rule when every nudge grazes.
// Bucket order in the reference is ascending triangle id; here buckets are
// unordered and "the first graze" is the graze with the smallest triangle id, so
// the partial heights are exactly the crossings of smaller ids.
#include <cuda_runtime.h>

#include <climits>

#include "cmg_device.cuh"
#include "cmg_exact.cuh"
#include "cmg_seg.cuh"
#include "cmg_types.h"
#include "cmg_util.h"
#include "engine_kernels.h"

namespace cmg::gpu {

namespace {

constexpr int kRowCols = 32;   // columns per CTA row segment
constexpr int kOccThreads = 128;
constexpr int kHCap = 32;      // crossings kept in shared memory per column
constexpr int kOccChunk = 4 * kOccThreads;  // bucket entries between two looks at the lists
constexpr int kOccQueue = 2 * kOccChunk;    // crossings and undecided entries waiting for FP64

__constant__ double c_nudge[6][2] = {
    {1.0e-6, 3.0e-7},  {-7.0e-7, 5.0e-7}, {4.0e-7, -9.0e-7},
    {-2.0e-6, -1.0e-6}, {8.0e-7, 6.0e-7}, {-5.0e-7, -4.0e-6},
};  // voxelize.cpp:148-151

__device__ __forceinline__ void load_tri(const double* __restrict__ soup, int64_t t, d3& a, d3& b,
                                         d3& c) {
    const double2* r = reinterpret_cast<const double2*>(soup + t * kSoupStride);
    double2 v0 = __ldg(r), v1 = __ldg(r + 1), v2 = __ldg(r + 2), v3 = __ldg(r + 3), v4 = __ldg(r + 4);
    a = {v0.x, v0.y, v1.x};
    b = {v1.y, v2.x, v2.y};
    c = {v3.x, v3.y, v4.x};
}

// plane_z (voxelize.cpp:107-114) in reference order.
__device__ __forceinline__ double plane_z(const d3& a, const d3& b, const d3& c, double x, double y) {
    double ux = dsub(b.x, a.x), uy = dsub(b.y, a.y), uz = dsub(b.z, a.z);
    double vx = dsub(c.x, a.x), vy = dsub(c.y, a.y), vz = dsub(c.z, a.z);
    double nx = dsub(dmul(uy, vz), dmul(uz, vy));
    double ny = dsub(dmul(uz, vx), dmul(ux, vz));
    double nz = dsub(dmul(ux, vy), dmul(uy, vx));
    return dsub(a.z, ddiv(dadd(dmul(nx, dsub(x, a.x)), dmul(ny, dsub(y, a.y))), nz));
}

// Sign of orient3d under the chosen semantics. FULL=false: returns 2 when the
// rounded determinant does not decide (COMPAT: it is exactly zero; EXACT: it is
// within the error bound). FULL=true: falls back to exact arithmetic.
template <bool FULL, int MODE>
__device__ __forceinline__ int o3d_sign(const d3& a, const d3& b, const d3& c, const d3& d,
                                        unsigned* exact_calls) {
    double perm;
    double det = o3d_fast(a, b, c, d, MODE == kPredExact ? &perm : nullptr);
    bool decided;
    if (MODE == kPredCompat) decided = det != 0.0;
    else decided = det > kO3dErrA * perm || -det > kO3dErrA * perm;
    if (decided) return sgn(det);
    if (!FULL) return 2;
    ++*exact_calls;
    return exact::orient3d_sign(a, b, c, d);
}

// One bucket triangle against the vertical segment P..Q (voxelize.cpp:127-141).
// Returns 0: no crossing, 1: crossing (height in *h), 2: graze (FULL) or
// undecided (filter).
template <bool FULL, int MODE>
__device__ __forceinline__ int column_tri(const d3& P, const d3& Q, const d3& a, const d3& b,
                                          const d3& c, double* h, unsigned* exact_calls,
                                          unsigned* orients = nullptr) {
    int sa = o3d_sign<FULL, MODE>(P, a, b, c, exact_calls);
    if (sa == 2 || sa == 0) return 2;
    int sb = o3d_sign<FULL, MODE>(Q, a, b, c, exact_calls);
    if (sb == 2 || sb == 0) return 2;
    if (orients) *orients += 2;
    if (sa == sb) return 0;
    if (orients) *orients += 3;
    int s1 = o3d_sign<FULL, MODE>(P, Q, a, b, exact_calls);
    if (s1 == 2 || s1 == 0) return 2;
    int s2 = o3d_sign<FULL, MODE>(P, Q, b, c, exact_calls);
    if (s2 == 2 || s2 == 0) return 2;
    int s3 = o3d_sign<FULL, MODE>(P, Q, c, a, exact_calls);
    if (s3 == 2 || s3 == 0) return 2;
    if (s1 != s2 || s2 != s3) return 0;
    *h = plane_z(a, b, c, P.x, P.y);
    return 1;
}

// Number of cell centres strictly below h: #{k : zc_k < h}. zc_k is non-decreasing in k,
// so {k : zc_k < h} is a prefix [0, n). n is guessed by one product and taken when the two
// centres about it agree; a search finds it otherwise.
__device__ __forceinline__ int centres_below(double hgt, double cz, double sp, double inv, int nz) {
    const int n = min(max(__double2int_rd(fma(dsub(hgt, cz), inv, 0.5)), 0), nz);
    int lo = 0, hi = nz;
    if (n == 0 || cell_center(cz, n - 1, sp) < hgt) lo = n;
    if (n == nz || !(cell_center(cz, n, sp) < hgt)) hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (cell_center(cz, mid, sp) < hgt) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The triangle's FP32 record for the segment test (three float4, lengths times the frame's
// s, a's xy offsets (dx, dy) from the grid's corner):
//   0: a.x, a.y, a.z - zmin, zmax - a.z
//   1: b - a, E2      2: c - a, E3
// each a FP64 difference rounded once (relative error u = 2^-24; zmax - a.z by one more
// difference). With p = (px, py) a column's offset, q = a - p, M >= |a.x|, |a.y|, |px|,
// |py|, T >= |x, y of b - a, c - a|, Z >= |z of them| and H >= |a.z - zmin|, |zmax - a.z|,
// to first order in u:
//   |q error| <= 4uM, so cross(q, b - a) is off by <= 20uMT and
//   cross(b - p, c - b) by <= 56uMT + 24uT^2;
//   n = (b - a) x (c - a): nx, ny off by <= 8uTZ, nz by <= 8uT^2, so
//   n.(P - a) and n.(Q - a) are off by <= 72uMTZ + 22uT^2H.
// Each FP64 determinant of the reference's order is off by at most 7.8e-16 of its
// permanent, which is <= 6 D^2 H with D = 2(M + T) and H over all height differences; the
// edges' determinants are cross * (zmax - zmin). E2 and E3 are above these sums, so a
// value beyond its bound has the sign that the rounded determinant has, and in the exact
// mode twice the bound (hence 2e-14) leaves it decided. Anything outside the range where
// no product over- or underflows gets an infinite bound; NaNs pass no comparison.
__device__ __forceinline__ void occ_record(const GridDesc& g, const OccFrame& f, const double* v,
                                           float dx, float dy, float4* r) {
    const float ax = dx * f.s, ay = dy * f.s;
    const float az = static_cast<float>(dsub(v[2], f.zmin)) * f.s;
    const float top = static_cast<float>(dsub(f.zmax, f.zmin)) * f.s;
    const float bz = top - az;
    float e[6];
    for (int k = 0; k < 6; ++k) e[k] = static_cast<float>(dsub(v[3 + k], v[k % 3])) * f.s;
    // the columns' centres, whose own rounding is a few ulps of the corner
    const float W = static_cast<float>(max(g.nx, g.ny)) * static_cast<float>(g.h) * f.s +
                    1e-15f * static_cast<float>(fmax(fabs(g.corner[0]), fabs(g.corner[1]))) * f.s;
    const float M = fmaxf(fmaxf(fabsf(ax), fabsf(ay)), W);
    const float T = fmaxf(fmaxf(fabsf(e[0]), fabsf(e[1])), fmaxf(fabsf(e[3]), fabsf(e[4])));
    const float Z = fmaxf(fabsf(e[2]), fabsf(e[5]));
    const float H = fabsf(az) + fabsf(bz) + Z;
    const float sum = ax + ay + az + bz + W + ((e[0] + e[1]) + (e[2] + e[3])) + (e[4] + e[5]);
    const float D = 2.0f * (M + T);
    float E2 = 4e-6f * (M + T) * T + 2e-14f * D * D * (H / top);
    float E3 = 6e-6f * M * T * Z + 2e-6f * T * T * H + 2e-14f * D * D * H;
    if (!(M <= 1e8f && T >= 1e-8f && T <= 1e8f && Z <= 1e8f && H <= 1e8f && top >= 1e-8f) ||
        sum != sum)
        E2 = E3 = __int_as_float(0x7f800000);
    r[0] = make_float4(ax, ay, az, bz);
    r[1] = make_float4(e[0], e[1], e[2], E2);
    r[2] = make_float4(e[3], e[4], e[5], E3);
}

// The segment over column offset (px, py) against a record: 0 no crossing, 1 a crossing,
// 2 not decided. The first two are the outcome of column_tri, with its count of orient3d.
__device__ __forceinline__ int column_tri32(const float4& r0, const float4& r1, const float4& r2,
                                            float px, float py, unsigned* orients) {
    const float qx = r0.x - px, qy = r0.y - py;
    const float nx = r1.y * r2.z - r1.z * r2.y;
    const float ny = r1.z * r2.x - r1.x * r2.z;
    const float nz = r1.x * r2.y - r1.y * r2.x;
    const float s = nx * qx + ny * qy;
    const float lo = s + nz * r0.z;   // -n.(P - a)
    const float hi = s - nz * r0.w;   // -n.(Q - a)
    if (!(fabsf(lo) > r2.w && fabsf(hi) > r2.w)) return 2;
    if ((lo > 0.0f) == (hi > 0.0f)) {
        *orients += 2;
        return 0;
    }
    const float fx = r2.x - r1.x, fy = r2.y - r1.y;   // c - b
    const float gx = qx + r1.x, gy = qy + r1.y;       // b - p
    const float ab = qx * r1.y - qy * r1.x;
    const float bc = gx * fy - gy * fx;
    const float ca = qy * r2.x - qx * r2.y;
    if (!(fminf(fabsf(ab), fminf(fabsf(bc), fabsf(ca))) > r1.w)) return 2;
    *orients += 5;
    return (ab > 0.0f) == (bc > 0.0f) && (bc > 0.0f) == (ca > 0.0f);
}

// cell_clamped by one FP32 product where that decides: the product is within 2^-22 of the
// quotient, relatively, so away from the whole numbers by more both have one floor.
// d32: the offset from the corner. (k_tri_prep for 262k triangles: 41 us with six
// FP64 divisions each; 19 us with these products and the record below, a store of 48 bytes.)
__device__ __forceinline__ int cell_of(double x, double corner, double h, float inv, int n, float* d32) {
    const float d = static_cast<float>(dsub(x, corner));
    *d32 = d;
    const float q = d * inv, f = floorf(q);
    const float r = q - f, m = 3e-7f * fabsf(q);
    if (!(inv > 0.0f && r > m && 1.0f - r > m)) return cell_clamped(x, corner, h, n);
    return f < 0.0f ? 0 : min(__float2int_rz(f), n - 1);
}

__global__ void k_tri_prep(const MeshSeg* __restrict__ segs, int nseg, int64_t ntris,
                           const double* __restrict__ pts, const int* __restrict__ tris,
                           double* __restrict__ soup, float4* __restrict__ otri,
                           int4* __restrict__ xybox, int64_t* __restrict__ pairs) {
    int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    const MeshSeg& s = segs[find_seg<&MeshSeg::tri_begin>(segs, nseg, t)];
    double v[9];
    for (int k = 0; k < 3; ++k) {
        int64_t vi = tris[3 * t + k];
        v[3 * k] = pts[3 * vi];
        v[3 * k + 1] = pts[3 * vi + 1];
        v[3 * k + 2] = pts[3 * vi + 2];
    }
    double2* r = reinterpret_cast<double2*>(soup + t * kSoupStride);
    r[0] = make_double2(v[0], v[1]);
    r[1] = make_double2(v[2], v[3]);
    r[2] = make_double2(v[4], v[5]);
    r[3] = make_double2(v[6], v[7]);
    r[4] = make_double2(v[8], 0.0);
    int i0 = s.g.nx, i1 = 0, j0 = s.g.ny, j1 = 0;
    float dx = 0.0f, dy = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float d0, d1;
        int i = cell_of(v[3 * k], s.g.corner[0], s.g.h, s.f.inv32, s.g.nx, &d0);
        int j = cell_of(v[3 * k + 1], s.g.corner[1], s.g.h, s.f.inv32, s.g.ny, &d1);
        if (k == 0) {
            dx = d0;
            dy = d1;
        }
        i0 = min(i0, i); i1 = max(i1, i);
        j0 = min(j0, j); j1 = max(j1, j);
    }
    if (otri) occ_record(s.g, s.f, v, dx, dy, otri + 3 * t);
    xybox[t] = make_int4(i0, i1, j0, j1);
    pairs[t] = static_cast<int64_t>(i1 - i0 + 1) * (j1 - j0 + 1);
}

// FILL=false: count bucket sizes into the zeroed colcnt; FILL=true: write bucket entries,
// taking the counts down to zero again. More than cap pairs: nothing (st->pairs says so).
// A warp finds its first pair's triangle together: with a binary search per pair, 29 + 27 us
// for 2.4M pairs of 262k triangles, 195 + 94 us for a batch of 24; now 18 + 18 and 75 + 66 us.
template <bool FILL>
__global__ void k_col_pairs(const MeshSeg* __restrict__ segs, int nseg, int64_t ntris,
                            const int4* __restrict__ xybox, const int64_t* __restrict__ pair_off,
                            int* __restrict__ colcnt, const int64_t* __restrict__ col_off,
                            int* __restrict__ col_list, int64_t cap, Stats* __restrict__ st,
                            unsigned long long* __restrict__ queue) {
    const int64_t npairs = pair_off[ntris];
    if (FILL && blockIdx.x == 0 && threadIdx.x == 0) {
        st->pairs = static_cast<unsigned long long>(npairs);
        if (npairs > cap && queue) atomicMax(queue, kQueueClosed);
    }
    if (npairs > cap) return;
    const int lane = threadIdx.x & 31;
    for (int64_t p0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31); p0 < npairs;
         p0 += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        // the last triangle at or before the warp's first pair, 33 intervals a step
        int64_t t0 = 0, len = ntris;  // t0 <= it < t0 + len
        while (len > 1) {
            const int64_t w = (len + 32) / 33, at = (lane + 1) * w;
            const int below = __popc(__ballot_sync(0xffffffffu, at < len && pair_off[t0 + at] <= p0));
            t0 += below * w;
            len = min(w, len - below * w);
        }
        // every triangle has a pair, so this warp's lie in the 32 from there
        const int64_t e = t0 + 1 + lane;
        const int64_t end = e < ntris ? pair_off[e] : INT64_MAX;
        const int64_t p = p0 + lane;
        int k = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1)
            if (__shfl_sync(0xffffffffu, end, k + st - 1) <= p) k += st;
        if (p >= npairs) continue;
        const int64_t t = t0 + k;
        const MeshSeg& s = segs[find_seg<&MeshSeg::tri_begin>(segs, nseg, t)];
        int4 bx = xybox[t];
        int64_t local = p - pair_off[t];
        int w = bx.y - bx.x + 1;
        int i = bx.x + static_cast<int>(local % w);
        int j = bx.z + static_cast<int>(local / w);
        int64_t col = s.col_begin + static_cast<int64_t>(j) * s.g.nx + i;
        if (FILL) col_list[col_off[col] + atomicSub(&colcnt[col], 1) - 1] = static_cast<int>(t);
        else atomicAdd(&colcnt[col], 1);
    }
}

// otri == nullptr: no records were made, and every entry is decided in FP64. xyz: the cells
// of one mesh's whole grid in [x][y][z] order.
//
// A column's entries decide 2 to 5 determinants each, and one warp instruction takes the
// FP64 pipe 16 cycles: deciding them all in FP64, with a column's few entries in a warp,
// took 770 us for 2.4M entries (262k triangles, 258 x 258 columns; the pipe 84 % busy, 15
// lanes of 32 in use). FP32 certifies all but about 1 % of them, the lanes run over the
// row's entries regardless of the column, and what needs FP64 (the crossings' heights, the
// undecided) waits for full warps: 120 us; 61 us with the crossings' layers stored so that
// neighbouring columns lie in different banks (layers [slot][column], one word of padding).
template <int MODE>
__global__ void __launch_bounds__(kOccThreads)
k_occ_filter(const MeshSeg* __restrict__ segs, int nseg, const double* __restrict__ soup,
             const float4* __restrict__ otri, const int64_t* __restrict__ col_off,
             const int* __restrict__ col_list, uint8_t* __restrict__ occ, bool xyz,
             int64_t* __restrict__ flagged, int64_t cap, Stats* __restrict__ st) {
    __shared__ int64_t off[kRowCols + 1];
    __shared__ float px[kRowCols];
    __shared__ int nbelow[kHCap][kRowCols + 1];
    __shared__ int hcnt[kRowCols];
    __shared__ int cflag[kRowCols];
    // entries waiting for FP64: certified crossings from the front, undecided ones from the
    // back, so that the warps of each list take one path
    __shared__ int qtri[kOccQueue];
    __shared__ uint8_t qcol[kOccQueue];
    __shared__ int qcross, qopen;
    if (static_cast<int64_t>(st->pairs) > cap) return;  // the buckets were not written

    const int64_t row = blockIdx.x;
    const int si = find_seg<&MeshSeg::row_begin>(segs, nseg, row);
    const MeshSeg& s = segs[si];
    const GridDesc g = s.g;
    const int rows_per_j = (g.nx + kRowCols - 1) / kRowCols;
    const int64_t lrow = row - s.row_begin;
    const int j = static_cast<int>(lrow / rows_per_j);
    const int i0 = static_cast<int>(lrow % rows_per_j) * kRowCols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t col0 = s.col_begin + static_cast<int64_t>(j) * g.nx + i0;
    const OccFrame fr = s.f;
    const double cy = cell_center(g.corner[1], j, g.h);
    const float py = static_cast<float>(dsub(cy, g.corner[1])) * fr.s;
    if (threadIdx.x <= kRowCols) off[threadIdx.x] = col_off[col0 + min(static_cast<int>(threadIdx.x), g.nx - i0)];
    if (threadIdx.x < kRowCols) {
        hcnt[threadIdx.x] = 0;
        cflag[threadIdx.x] = 0;
        px[threadIdx.x] =
            static_cast<float>(dsub(cell_center(g.corner[0], i0 + threadIdx.x, g.h), g.corner[0])) * fr.s;
    }
    if (threadIdx.x == 0) qcross = qopen = 0;
    __syncthreads();

    unsigned dummy = 0, orients = 0, crossings = 0;
    const auto height = [&](int c, double hgt) {
        ++crossings;
        const int slot = atomicAdd(&hcnt[c], 1);
        if (slot < kHCap) nbelow[slot][c] = centres_below(hgt, g.corner[2], g.h, fr.inv, g.nz);
        else cflag[c] = 1;
    };
    const int64_t end = off[kRowCols];
    for (int64_t base = off[0]; base < end; base += kOccChunk) {
#pragma unroll
        for (int u = 0; u < kOccChunk / kOccThreads; ++u) {
            const int64_t e = base + u * kOccThreads + threadIdx.x;
            if (e >= end) continue;
            const int t = col_list[e];
            int c = 0;
#pragma unroll
            for (int w = kRowCols / 2; w > 0; w >>= 1)
                if (off[c + w] <= e) c += w;
            int r = 2;
            if (otri) {
                const float4* rec = otri + 3 * static_cast<int64_t>(t);
                r = column_tri32(__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), px[c], py, &orients);
            }
            if (r) {
                const int q = r == 1 ? atomicAdd(&qcross, 1) : kOccQueue - 1 - atomicAdd(&qopen, 1);
                qtri[q] = t;
                qcol[q] = static_cast<uint8_t>(c);
            }
        }
        __syncthreads();
        const int nc = qcross, no = qopen;
        __syncthreads();
        if (nc + no <= kOccQueue - kOccChunk && base + kOccChunk < end) continue;
        for (int q = threadIdx.x; q < nc; q += kOccThreads) {
            d3 a, b, cc;
            load_tri(soup, qtri[q], a, b, cc);
            const int c = qcol[q];
            height(c, plane_z(a, b, cc, cell_center(g.corner[0], i0 + c, g.h), cy));
        }
        for (int q = threadIdx.x; q < no; q += kOccThreads) {
            d3 a, b, cc;
            load_tri(soup, qtri[kOccQueue - 1 - q], a, b, cc);
            const int c = qcol[kOccQueue - 1 - q];
            const double cx = cell_center(g.corner[0], i0 + c, g.h);
            double hgt;
            const int r = column_tri<false, MODE>({cx, cy, fr.zmin}, {cx, cy, fr.zmax}, a, b, cc, &hgt,
                                                  &dummy, &orients);
            if (r == 2) cflag[c] = 1;
            else if (r == 1) height(c, hgt);
        }
        __syncthreads();
        if (threadIdx.x == 0) qcross = qopen = 0;
        __syncthreads();
    }
    __syncthreads();
    // parity bytes of the slab [z0, z1) (the column spans the whole grid)
    if (xyz) {  // lane = layer, warps stride columns: a column's bytes are consecutive
        for (int c = warp; c < min(kRowCols, g.nx - i0); c += kOccThreads / 32) {
            if (cflag[c]) continue;
            const int m = hcnt[c];
            uint8_t* base = occ + (static_cast<int64_t>(i0 + c) * g.ny + j) * g.nz;
            for (int k = lane; k < g.nz; k += 32) {
                int par = 0;
                for (int q = 0; q < m; ++q) par ^= (nbelow[q][c] > k);
                base[k] = static_cast<uint8_t>(par);
            }
        }
    } else {  // lane = column, warps stride k: one warp writes 32 consecutive bytes
        const int c = lane, i = i0 + lane;
        const bool live = i < g.nx && !cflag[c];
        const int m = min(hcnt[c], kHCap);
        uint8_t* base = occ + s.vox_begin + static_cast<int64_t>(j) * g.nx + i;
        const int64_t kstride = static_cast<int64_t>(g.nx) * g.ny;
        for (int k = g.z0 + warp; k < g.z1; k += kOccThreads / 32) {
            if (!live) continue;
            int par = 0;
            for (int q = 0; q < m; ++q) par ^= (nbelow[q][c] > k);
            base[(k - g.z0) * kstride] = static_cast<uint8_t>(par);
        }
    }
    {
        long long o = warp_sum(static_cast<long long>(orients));
        long long x = warp_sum(static_cast<long long>(crossings));
        if (lane == 0 && o) atomicAdd(&st->orient_calls, static_cast<unsigned long long>(o));
        if (lane == 0 && x) atomicAdd(&st->crossings, static_cast<unsigned long long>(x));
    }
    if (warp == 0) {
        const int i = i0 + lane;
        bool f = i < g.nx && cflag[lane];
        unsigned mask = __ballot_sync(0xffffffffu, f);
        int n = __popc(mask);
        unsigned long long base = 0;
        if (lane == 0 && n) base = atomicAdd(&st->flagged_columns, static_cast<unsigned long long>(n));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (f) {
            int rank = __popc(mask & ((1u << lane) - 1u));
            flagged[base + rank] = s.col_begin + static_cast<int64_t>(j) * g.nx + i;
        }
    }
}

// One warp per listed column (grid-stride); scratch hs[e] holds the crossing height
// of bucket entry e (NaN-free flag in hv[e]) of the attempt being kept.
template <int MODE>
__global__ void __launch_bounds__(128)
k_occ_exact(const MeshSeg* __restrict__ segs, int nseg, const double* __restrict__ soup,
            const int64_t* __restrict__ col_off, const int* __restrict__ col_list,
            const int64_t* __restrict__ flagged, double* __restrict__ hs, uint8_t* __restrict__ hv,
            uint8_t* __restrict__ occ, bool xyz, Stats* __restrict__ st) {
    const int lane = threadIdx.x & 31;
    const int64_t nflag = static_cast<int64_t>(st->flagged_columns);
    const int64_t wstride = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
    for (int64_t w = static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5);
         w < nflag; w += wstride) {
        const int64_t col = flagged[w];
        const int si = find_seg<&MeshSeg::col_begin>(segs, nseg, col);
        const MeshSeg& s = segs[si];
        const GridDesc g = s.g;
        const int64_t lc = col - s.col_begin;
        const int i = static_cast<int>(lc % g.nx), j = static_cast<int>(lc / g.nx);
        const double zmin = dsub(g.corner[2], g.h);
        const double zmax = dadd(g.corner[2], dmul(static_cast<double>(g.nz + 1), g.h));
        const double cx = cell_center(g.corner[0], i, g.h);
        const double cy = cell_center(g.corner[1], j, g.h);
        const int64_t e0 = col_off[col], e1 = col_off[col + 1];
        unsigned exact_calls = 0;
        int limit = INT_MAX;  // crossings of triangles with id < limit are kept
        for (int attempt = 0; attempt < 7; ++attempt) {
            double x = cx, y = cy;
            if (attempt > 0) {
                x = dadd(cx, dmul(c_nudge[attempt - 1][0], g.h));
                y = dadd(cy, dmul(c_nudge[attempt - 1][1], g.h));
            }
            const d3 P{x, y, zmin}, Q{x, y, zmax};
            int first_graze = INT_MAX;
            for (int64_t e = e0 + lane; e < e1; e += 32) {
                d3 a, b, cc;
                const int t = col_list[e];
                load_tri(soup, t, a, b, cc);
                double hgt = 0.0;
                int r = column_tri<true, MODE>(P, Q, a, b, cc, &hgt, &exact_calls);
                if (r == 2) first_graze = min(first_graze, t);
                hs[e] = hgt;
                hv[e] = static_cast<uint8_t>(r == 1);
            }
            first_graze = warp_min(first_graze);
            if (first_graze == INT_MAX) {
                limit = INT_MAX;
                if (attempt > 0 && lane == 0) atomicAdd(&st->nudged_columns, 1ull);
                break;
            }
            limit = first_graze;  // if this is the last attempt, its partial result stays
            if (attempt == 6 && lane == 0) {
                atomicAdd(&st->nudged_columns, 1ull);
                atomicAdd(&st->exhausted_columns, 1ull);
            }
        }
        __syncwarp();
        long long ec = warp_sum(static_cast<long long>(exact_calls));
        if (lane == 0 && ec) atomicAdd(&st->exact_calls, static_cast<unsigned long long>(ec));
        // parity per cell: crossings of ids < limit strictly above the cell centre
        uint8_t* base = xyz ? occ + (static_cast<int64_t>(i) * g.ny + j) * g.nz
                            : occ + s.vox_begin + static_cast<int64_t>(j) * g.nx + i;
        const int64_t kstride = xyz ? 1 : static_cast<int64_t>(g.nx) * g.ny;
        for (int k = g.z0 + lane; k < g.z1; k += 32) {  // the slab's layers
            const double zc = cell_center(g.corner[2], k, g.h);
            int par = 0;
            for (int64_t e = e0; e < e1; ++e)
                if (hv[e] && col_list[e] < limit && hs[e] > zc) par ^= 1;
            base[(k - g.z0) * kstride] = static_cast<uint8_t>(par);
        }
    }
}

}  // namespace

void launch_tri_prep(const MeshSeg* segs, int nseg, int64_t ntris, const double* pts,
                     const int* tris, double* soup, float4* otri, int4* xybox, int64_t* pairs,
                     cudaStream_t st) {
    if (ntris == 0) return;
    k_tri_prep<<<static_cast<unsigned>((ntris + 255) / 256), 256, 0, st>>>(
        segs, nseg, ntris, pts, tris, soup, otri, xybox, pairs);
    CMG_LAUNCH();
}

void launch_col_pairs(bool fill, const MeshSeg* segs, int nseg, int64_t ntris, const int4* xybox,
                      const int64_t* pair_off, int* colcnt, const int64_t* col_off, int* col_list,
                      int64_t cap, Stats* stats, unsigned long long* queue, int grid, cudaStream_t st) {
    if (ntris == 0) return;
    if (fill)
        k_col_pairs<true><<<grid, 256, 0, st>>>(segs, nseg, ntris, xybox, pair_off, colcnt, col_off,
                                                col_list, cap, stats, queue);
    else
        k_col_pairs<false><<<grid, 256, 0, st>>>(segs, nseg, ntris, xybox, pair_off, colcnt, col_off,
                                                 col_list, cap, stats, queue);
    CMG_LAUNCH();
}

void launch_occ_filter(int mode, const MeshSeg* segs, int nseg, int64_t nrows, const double* soup,
                       const float4* otri, const int64_t* col_off, const int* col_list, uint8_t* occ,
                       bool xyz, int64_t* flagged,
                       int64_t cap, Stats* stats, cudaStream_t st) {
    if (nrows == 0) return;
    if (mode == kPredExact)
        k_occ_filter<kPredExact><<<static_cast<unsigned>(nrows), kOccThreads, 0, st>>>(
            segs, nseg, soup, otri, col_off, col_list, occ, xyz, flagged, cap, stats);
    else
        k_occ_filter<kPredCompat><<<static_cast<unsigned>(nrows), kOccThreads, 0, st>>>(
            segs, nseg, soup, otri, col_off, col_list, occ, xyz, flagged, cap, stats);
    CMG_LAUNCH();
}

void launch_occ_exact(int mode, const MeshSeg* segs, int nseg, const double* soup,
                      const int64_t* col_off, const int* col_list, const int64_t* flagged,
                      double* hs, uint8_t* hv, uint8_t* occ, bool xyz, Stats* stats, int grid,
                      cudaStream_t st) {
    if (mode == kPredExact)
        k_occ_exact<kPredExact><<<grid, 128, 0, st>>>(segs, nseg, soup, col_off, col_list, flagged,
                                                      hs, hv, occ, xyz, stats);
    else
        k_occ_exact<kPredCompat><<<grid, 128, 0, st>>>(segs, nseg, soup, col_off, col_list, flagged,
                                                       hs, hv, occ, xyz, stats);
    CMG_LAUNCH();
}

int occ_row_cols() { return kRowCols; }

}  // namespace cmg::gpu
