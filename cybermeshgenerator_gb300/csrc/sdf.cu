// sdf.cu — signed distance field: nearest boundary triangle per cell.
//
// The reference computes, per cell centre, the minimum of point_tri_dist2
// (Ericson, src/voxelize/voxelize.cpp:202-247) over the triangles found by a
// Chebyshev ring search of 3-D buckets (:251-326); its pruning is exact, so the
// result equals the brute-force minimum over all triangles. Here:
//
//   k_sdf_tri_prep   centroid c_t, radius e_t = max |v - c_t| (rounded up), bin of
//                    c_t in the brick grid; triangles larger than two bricks (or
//                    degenerate) go to a per-mesh "always considered" list
//   k_bin_fill       bin -> triangle CSR, the entries' centroids and radii in its order;
//                    k_bin_balls: a ball around each bin's triangles
//   k_brick_walk     one to eight warps per brick: a ring walk over bins gives an upper
//                    bound U on the distance from the brick centre to the surface, then
//                    the candidate list = every triangle whose lower bound
//                    |c - c_t| - e_t - r_B can be <= U + r_B (r_B = brick radius) and that
//                    the box test around the nearest centroid leaves, with margins far
//                    above FP32 and FP64 rounding
// and the lists are evaluated by warps of 4^3 cells (sdf_near.cu; plain FP64: sdf_sub.cu),
// or at brick edges 4 and 8 by
//   k_sdf_fp64       one CTA per brick, candidates staged through shared memory;
//                    each thread owns voxels and evaluates Ericson in the reference
//                    operation order (FP64, no FMA): bit-identical to the reference
//   k_sdf_mixed      same walk in FP32 on brick-recentred coordinates (normals from
//                    FP64) with a stated error bound; cells within a band of the
//                    surface are re-evaluated in FP64 over the candidates whose
//                    FP32 distance is within twice the bound of the best, which
//                    reproduces the FP64 minimum exactly there.
// Both evaluation kernels skip a candidate for a whole warp when no lane's cells
// can reach it (bounding sphere of the triangle vs the current best).
#include <cuda_runtime.h>

#include <cfloat>
#include <climits>

#include "cmg_device.cuh"
#include "cmg_sdf.cuh"
#include "cmg_seg.cuh"
#include "cmg_sub.cuh"
#include "cmg_types.h"
#include "cmg_util.h"
#include "engine_kernels.h"

namespace cmg::gpu {

namespace {

using namespace sdf;
static_assert(sizeof(TriRec) == kTriRecBytes, "the workspace carves kTriRecBytes per record");

__device__ __forceinline__ float round_up_f(double x) { return __double2float_ru(x); }

// ------------------------------------------------------------------ triangle prep
// tinfo (float4 per triangle): centroid relative to the mesh grid corner (FP32,
// nearest) and the radius e_t rounded up (plus the rounding of the centroid). tnorm, for the
// plain FP64 evaluation, may be null; tlo and thi are written for large triangles, the only
// ones whose boxes are read.
// 128k triangles: 320 us with one atomic per triangle on its mesh's largest radius (twice),
// coordinate scale and bin; 118 us with one per warp, bound by some 300 FP64 instructions a
// triangle on the narrow pipe (24 meshes: 677 -> 288 us, k_bin_fill 109 -> 12).
__global__ void k_sdf_tri_prep(const MeshSeg* __restrict__ segs, int nseg, int64_t ntris,
                               const double* __restrict__ pts, const int* __restrict__ tris,
                               float4* __restrict__ tinfo,
                               float4* __restrict__ tinfo_lo, TriRec* __restrict__ trec,
                               float4* __restrict__ tnorm,
                               float4* __restrict__ tlo, float4* __restrict__ thi,
                               int64_t* __restrict__ tbin, int* __restrict__ bincnt,
                               int* __restrict__ large_cnt, unsigned* __restrict__ emax_bits,
                               Stats* __restrict__ st) {
    int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    const int si = find_seg<&MeshSeg::tri_begin>(segs, nseg, t);
    const MeshSeg& s = segs[si];
    d3 a, b, c;
    {
        const double* pa = pts + 3 * static_cast<int64_t>(tris[3 * t]);
        const double* pb = pts + 3 * static_cast<int64_t>(tris[3 * t + 1]);
        const double* pc = pts + 3 * static_cast<int64_t>(tris[3 * t + 2]);
        a = {pa[0], pa[1], pa[2]};
        b = {pb[0], pb[1], pb[2]};
        c = {pc[0], pc[1], pc[2]};
    }
    const double* K = s.g.corner;
    // centroid in FP64 (any rounding is covered by the radius padding below)
    double cx = (a.x + b.x + c.x) / 3.0, cy = (a.y + b.y + c.y) / 3.0, cz = (a.z + b.z + c.z) / 3.0;
    double r2 = 0.0;
    const d3 V[3] = {a, b, c};
    for (int k = 0; k < 3; ++k) {
        double dx = V[k].x - cx, dy = V[k].y - cy, dz = V[k].z - cz;
        r2 = fmax(r2, dx * dx + dy * dy + dz * dz);
    }
    float4 ci, cl;
    split2(cx - K[0], ci.x, cl.x);
    split2(cy - K[1], ci.y, cl.y);
    split2(cz - K[2], ci.z, cl.z);
    cl.w = 0.f;
    tinfo_lo[t] = cl;
    // radius: sqrt rounded up, padded for the FP32 centroid (|err| <= u*|c - K|*sqrt3)
    double pad = 2.0 * kU32 * (fabs(cx - K[0]) + fabs(cy - K[1]) + fabs(cz - K[2])) + 1e-300;
    ci.w = round_up_f(sqrt(r2) * (1.0 + 1e-12) + pad);
    tinfo[t] = ci;
    // translation-invariant FP32 record (from FP64)
    double ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z;
    double vx = c.x - a.x, vy = c.y - a.y, vz = c.z - a.z;
    double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    bool degenerate = !(nx * nx + ny * ny + nz * nz > 0.0);
    bool thin;  // without a face in its FP32 record: the reference's distance may be none (NaN)
    {
        const double lu = sqrt(ux * ux + uy * uy + uz * uz), lv = sqrt(vx * vx + vy * vy + vz * vz);
        if (tnorm) {
            double nl = sqrt(nx * nx + ny * ny + nz * nz);
            double n3[3] = {0.0, 0.0, 0.0};
            if (nl > 0.0) { n3[0] = nx / nl; n3[1] = ny / nl; n3[2] = nz / nl; }
            // the FP64 path's plane bound: the unit normal in FP32 and a bound on its distance
            // from the exact one: the cross product of rounded edges errs by at most
            // 21 u |u| |v| (as a vector), which turns its direction by at most twice that
            // over |u x v|; then the normalisation and the FP32 rounding of the components
            const double en = nl > 0.0 ? 50.0 * kU64 * lu * lv / nl + 1.2e-7 : 0.0;
            tnorm[t] = make_float4(static_cast<float>(n3[0]), static_cast<float>(n3[1]),
                                   static_cast<float>(n3[2]), round_up_f(en));
        }
        // the mixed path's record in the triangle's frame: u along b - a (else along
        // c - a, else x), v from c - a by two Gram-Schmidt passes (so c = a + cx u +
        // cy v to FP64 rounding however thin the triangle), n = u x v
        double U[3], Vv[3], bx;
        const double lab = lu, lac = lv;
        if (lab > 0.0) { U[0] = ux / lab; U[1] = uy / lab; U[2] = uz / lab; bx = lab; }
        else if (lac > 0.0) { U[0] = vx / lac; U[1] = vy / lac; U[2] = vz / lac; bx = 0.0; }
        else { U[0] = 1.0; U[1] = 0.0; U[2] = 0.0; bx = 0.0; }
        double ccx = vx * U[0] + vy * U[1] + vz * U[2];
        double rx = vx - ccx * U[0], ry = vy - ccx * U[1], rz = vz - ccx * U[2];
        const double kk = rx * U[0] + ry * U[1] + rz * U[2];
        ccx += kk;
        rx -= kk * U[0]; ry -= kk * U[1]; rz -= kk * U[2];
        // a residual at the rounding level (exactly collinear vertices leave one along u)
        // carries no direction: the triangle is taken as collinear, which moves c by at
        // most 1e-9 of the triangle's size (far inside the stated FP32 error)
        double ccy = sqrt(rx * rx + ry * ry + rz * rz);
        if (!(ccy > 1e-9 * fmax(lab, lac))) ccy = 0.0;
        if (ccy > 0.0) {
            Vv[0] = rx / ccy; Vv[1] = ry / ccy; Vv[2] = rz / ccy;
        } else {
            // collinear: any unit vector across u (u x the axis least aligned with u)
            const int ax = fabs(U[0]) <= fabs(U[1]) && fabs(U[0]) <= fabs(U[2]) ? 0 : (fabs(U[1]) <= fabs(U[2]) ? 1 : 2);
            const double A[3] = {ax == 0 ? 1.0 : 0.0, ax == 1 ? 1.0 : 0.0, ax == 2 ? 1.0 : 0.0};
            double wx = A[1] * U[2] - A[2] * U[1], wy = A[2] * U[0] - A[0] * U[2], wz = A[0] * U[1] - A[1] * U[0];
            const double wl = sqrt(wx * wx + wy * wy + wz * wz);
            Vv[0] = wx / wl; Vv[1] = wy / wl; Vv[2] = wz / wl;
        }
        const double N[3] = {U[1] * Vv[2] - U[2] * Vv[1], U[2] * Vv[0] - U[0] * Vv[2], U[0] * Vv[1] - U[1] * Vv[0]};
        TriRec r;
        r.o0[0] = static_cast<float>(a.x - cx);
        r.o0[1] = static_cast<float>(a.y - cy);
        r.o0[2] = static_cast<float>(a.z - cz);
        for (int q = 0; q < 3; ++q) {
            r.nn[q] = static_cast<float>(N[q]);
            r.uu[q] = static_cast<float>(U[q]);
            r.vv[q] = static_cast<float>(Vv[q]);
        }
        // the triangle lies in the frame's plane (to FP64 rounding), every triangle has
        // one, and its FP32 normal is within the rounding of a unit vector (sqrt(3) u)
        r.nerr = kRecNormalErr;
        r.bx = static_cast<float>(bx);
        r.cx = static_cast<float>(ccx);
        r.cy = static_cast<float>(ccy);
        r.e1x = static_cast<float>(ccx - bx);
        r.ib = bx > 0.0 ? static_cast<float>(1.0 / bx) : 0.f;
        const double l1 = (ccx - bx) * (ccx - bx) + ccy * ccy, l2 = ccx * ccx + ccy * ccy;
        r.inv1 = l1 > 0.0 ? static_cast<float>(1.0 / l1) : 0.f;
        r.inv2 = l2 > 0.0 ? static_cast<float>(1.0 / l2) : 0.f;
        thin = !(bx > 0.0 && ccy > 0.0);
        r.ok = thin ? 0.f : 1.f;
        r.pad_[0] = r.pad_[1] = r.pad_[2] = 0.f;
        trec[t] = r;
    }
    // degenerate (zero-area), thin or larger than two bricks: always considered
    const double bw = static_cast<double>(s.brick) * s.g.h;
    const bool large = degenerate || thin || sqrt(r2) > 2.0 * bw;
    if (thin) atomicAdd(&st->thin, 1ull);
    // per segment, one set of atomics per warp: the mesh's coordinate scale max |v - K|
    // (rounded up) for the FP32 tolerances (k_seg_finish folds in the grid extent), the
    // largest radius of all its triangles (the mixed path's error bounds) and of the binned
    // ones, and the large ones' count
    {
        // (the largest by the bits, off the FP64 pipe; NaNs do not count)
        unsigned long long m = 0ull;
        auto most = [&](double v) {
            const unsigned long long w = static_cast<unsigned long long>(__double_as_longlong(fabs(v)));
            if (w > m && w <= 0x7ff0000000000000ull) m = w;
        };
        for (int k = 0; k < 3; ++k) {
            most(V[k].x - K[0]);
            most(V[k].y - K[1]);
            most(V[k].z - K[2]);
        }
        const unsigned bits = __float_as_uint(round_up_f(__longlong_as_double(static_cast<long long>(m))));
        const unsigned grp = __match_any_sync(__activemask(), si);
        const unsigned scale = __reduce_max_sync(grp, bits), w = __float_as_uint(ci.w);
        const unsigned all = __reduce_max_sync(grp, w), binned = __reduce_max_sync(grp, large ? 0u : w);
        const unsigned n = __reduce_add_sync(grp, large ? 1u : 0u);
        if ((threadIdx.x & 31) == __ffs(grp) - 1) {
            atomicMax(&emax_bits[nseg + si], scale);
            atomicMax(&emax_bits[2 * nseg + si], all);
            if (binned) atomicMax(&emax_bits[si], binned);
            if (n) atomicAdd(&large_cnt[si], static_cast<int>(n));
        }
    }
    if (large) {
        tlo[t] = make_float4(__double2float_rd(fmin(a.x, fmin(b.x, c.x)) - K[0]),
                             __double2float_rd(fmin(a.y, fmin(b.y, c.y)) - K[1]),
                             __double2float_rd(fmin(a.z, fmin(b.z, c.z)) - K[2]),
                             degenerate || thin ? 1.f : 0.f);
        thi[t] = make_float4(__double2float_ru(fmax(a.x, fmax(b.x, c.x)) - K[0]),
                             __double2float_ru(fmax(a.y, fmax(b.y, c.y)) - K[1]),
                             __double2float_ru(fmax(a.z, fmax(b.z, c.z)) - K[2]), 0.f);
        tbin[t] = -1;
        return;
    }
    // the bin of the centroid among the mesh's bricks (along z those of its slab, from
    // brick layer bzo), clamped: a clamped triangle lies outside the bins' box, and no
    // point inside the box is nearer its clamped position than its own
    // (an FP32 product decides where it is clear of the whole numbers by more than its error)
    const float inv = 1.f / static_cast<float>(bw);
    auto bin_of = [&](float d32, double d) {
        const float v = d32 * inv, f = floorf(v), rest = v - f, m = 4e-7f * fabsf(v);
        if (rest > m && 1.f - rest > m && fabsf(v) < 1e6f) return static_cast<int>(f);
        return static_cast<int>(floor(d / bw));
    };
    int bx = bin_of(ci.x, cx - K[0]);
    int by = bin_of(ci.y, cy - K[1]);
    int bz = bin_of(ci.z, cz - K[2]) - s.bzo;
    bx = min(max(bx, 0), s.bnx - 1);
    by = min(max(by, 0), s.bny - 1);
    bz = min(max(bz, 0), s.bnz - 1);
    int64_t bin = s.brick_begin + (static_cast<int64_t>(bz) * s.bny + by) * s.bnx + bx;
    tbin[t] = bin;
    // (neighbouring triangles share bins: one atomic per bin and warp, here and in k_bin_fill)
    const unsigned grp = __match_any_sync(__activemask(), bin);
    if ((threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&bincnt[bin], __popc(grp));
}

// Bin -> triangle CSR. bin_info: the triangles' tinfo in the list's order, so that the walks
// read the bins' entries in order and the ids only of those they take.
__global__ void k_bin_fill(int64_t ntris, const int64_t* __restrict__ tbin,
                           const int64_t* __restrict__ bin_off, int* __restrict__ bincur,
                           const float4* __restrict__ tinfo, int* __restrict__ bin_list,
                           float4* __restrict__ bin_info, const MeshSeg* __restrict__ segs, int nseg,
                           int* __restrict__ large_cur, int* __restrict__ large_list) {
    int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= ntris) return;
    const int lane = threadIdx.x & 31;
    int64_t b = tbin[t];
    if (b >= 0) {
        const unsigned grp = __match_any_sync(__activemask(), b);
        const int lead = __ffs(grp) - 1, n = __popc(grp);
        int left = 0;
        if (lane == lead) left = atomicSub(&bincur[b], n);  // the counts, taken down to zero
        left = __shfl_sync(grp, left, lead);
        const int64_t at = bin_off[b] + left - n + __popc(grp & ((1u << lane) - 1u));
        bin_list[at] = static_cast<int>(t);
        bin_info[at] = tinfo[t];
    } else {
        const int si = find_seg<&MeshSeg::tri_begin>(segs, nseg, t);
        int slot = atomicAdd(&large_cur[si], 1);
        large_list[segs[si].large_begin + slot] = static_cast<int>(t);
    }
}

// Per bin, a ball around its triangles: the middle of its centroids' box, the largest
// distance of a centroid from it (w; -1: an empty bin) and of a triangle (bin_reach), so
// that the walks skip whole bins. One warp per bin.
__global__ void k_bin_balls(int64_t nbins, const int64_t* __restrict__ bin_off,
                            const float4* __restrict__ bin_info, const MeshSeg* __restrict__ segs,
                            int nseg, float4* __restrict__ bin_ball, float* __restrict__ bin_reach) {
    const int64_t b = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (b >= nbins) return;
    const int64_t e0 = bin_off[b], e1 = bin_off[b + 1];
    if (e0 == e1) {
        if (lane == 0) bin_ball[b] = make_float4(0.f, 0.f, 0.f, -1.f);
        return;
    }
    float lx = FLT_MAX, ly = FLT_MAX, lz = FLT_MAX, hx = -FLT_MAX, hy = -FLT_MAX, hz = -FLT_MAX;
    // (the last entry again beyond the end: four loads in flight in long bins)
    for (int64_t e = e0 + lane; e - lane < e1; e += 128) {
        float4 t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = bin_info[min(e + 32 * j, e1 - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            lx = fminf(lx, t[j].x); ly = fminf(ly, t[j].y); lz = fminf(lz, t[j].z);
            hx = fmaxf(hx, t[j].x); hy = fmaxf(hy, t[j].y); hz = fmaxf(hz, t[j].z);
        }
    }
    const float cx = 0.5f * (warp_min(lx) - warp_min(-hx)), cy = 0.5f * (warp_min(ly) - warp_min(-hy)),
                cz = 0.5f * (warp_min(lz) - warp_min(-hz));
    float rc = 0.f, rt = 0.f;
    for (int64_t e = e0 + lane; e - lane < e1; e += 128) {
        float4 t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = bin_info[min(e + 32 * j, e1 - 1)];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float dx = t[j].x - cx, dy = t[j].y - cy, dz = t[j].z - cz;
            const float d = sqrtf(dx * dx + dy * dy + dz * dz);
            rc = fmaxf(rc, d);
            rt = fmaxf(rt, d + t[j].w);
        }
    }
    rc = -warp_min(-rc);
    rt = -warp_min(-rt);
    if (lane == 0) {
        const float tol = list_tol(segs[find_seg<&MeshSeg::brick_begin>(segs, nseg, b)].scale);
        bin_ball[b] = make_float4(cx, cy, cz, rc * (1.f + 8.f * kU32) + tol);
        bin_reach[b] = rt * (1.f + 8.f * kU32) + tol;
    }
}

// Scans the meshes' always-considered counts (one block) and writes each mesh's range, emax and coordinate scale (the
// larger of max |v - K| over its points and the grid extent, with 1e-4 slack)
// into its segment.
constexpr int kSegThreads = 128;
__global__ void __launch_bounds__(kSegThreads) k_seg_finish(MeshSeg* segs, int nseg, const int* __restrict__ large_cnt,
                                                            const unsigned* __restrict__ emax_bits) {
    __shared__ int64_t s_w[kSegThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t carry = 0;
    for (int i0 = 0; i0 < nseg; i0 += kSegThreads) {
        const int i = i0 + threadIdx.x;
        const int64_t n = i < nseg ? large_cnt[i] : 0;
        int64_t end = n;  // inclusive prefix
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += y;
        }
        if (lane == 31) s_w[warp] = end;
        __syncthreads();
        int64_t total = 0;
#pragma unroll
        for (int w = 0; w < kSegThreads / 32; ++w) {
            if (w < warp) end += s_w[w];
            total += s_w[w];
        }
        __syncthreads();
        end += carry;
        carry += total;
        if (i >= nseg) continue;
        segs[i].large_begin = end - n;
        segs[i].large_end = end;
        segs[i].emax = __uint_as_float(emax_bits[i]);
        segs[i].emax_all = __uint_as_float(emax_bits[2 * nseg + i]);
        const GridDesc& g = segs[i].g;
        const double ext = g.h * static_cast<double>(max(g.nx, max(g.ny, g.nz)));
        const double sc = fmax(static_cast<double>(__uint_as_float(emax_bits[nseg + i])), ext);
        segs[i].scale = __double2float_ru(sc * 1.0001);
    }
}

// ------------------------------------------------------------------ brick geometry
struct BrickGeo {
    int bx, by, bz;
    int x0, y0, z0, x1, y1, z1;  // cell range [x0, x1)
    float cx, cy, cz;            // centre of the cell-centre box, relative to the corner
    float rb;                    // half-diagonal of that box (rounded up)
};

__device__ __forceinline__ BrickGeo brick_geo(const MeshSeg& s, int64_t lb) {
    BrickGeo q;
    q.bx = static_cast<int>(lb % s.bnx);
    q.by = static_cast<int>((lb / s.bnx) % s.bny);
    q.bz = static_cast<int>(lb / (static_cast<int64_t>(s.bnx) * s.bny));
    const int B = s.brick;
    q.x0 = q.bx * B; q.x1 = min(q.x0 + B, s.g.nx);
    q.y0 = q.by * B; q.y1 = min(q.y0 + B, s.g.ny);
    q.z0 = (q.bz + s.bzo) * B; q.z1 = min(q.z0 + B, s.g.nz);  // bz counts from the slab's bricks
    const float h = static_cast<float>(s.g.h);
    q.cx = span_centre(q.x0, q.x1, h);
    q.cy = span_centre(q.y0, q.y1, h);
    q.cz = span_centre(q.z0, q.z1, h);
    double hx = 0.5 * (q.x1 - q.x0 - 1) * s.g.h, hy = 0.5 * (q.y1 - q.y0 - 1) * s.g.h,
           hz = 0.5 * (q.z1 - q.z0 - 1) * s.g.h;
    q.rb = __double2float_ru(sqrt(hx * hx + hy * hy + hz * hz) * (1.0 + 1e-9));
    return q;
}

// Shell q of Chebyshev radius r -> offset (dx, dy, dz).
__device__ __forceinline__ void shell_offset(int r, int q, int& dx, int& dy, int& dz) {
    if (r == 0) { dx = dy = dz = 0; return; }
    const int w = 2 * r + 1, v = 2 * r - 1;
    const int A = w * w, Bn = w * v;
    if (q < 2 * A) {
        dz = (q / A) ? r : -r;
        int rem = q % A;
        dy = rem / w - r;
        dx = rem % w - r;
        return;
    }
    q -= 2 * A;
    if (q < 2 * Bn) {
        dy = (q / Bn) ? r : -r;
        int rem = q % Bn;
        dz = rem / w - (r - 1);
        dx = rem % w - r;
        return;
    }
    q -= 2 * Bn;
    const int C = v * v;
    dx = (q / C) ? r : -r;
    int rem = q % C;
    dz = rem / v - (r - 1);
    dy = rem % v - (r - 1);
}

__device__ __forceinline__ int shell_count(int r) { return r == 0 ? 1 : 24 * r * r + 2; }

// Bin k of the Chebyshev shell r around the brick, or -1 (not in the grid).
__device__ __forceinline__ int64_t shell_bin(const MeshSeg& s, const BrickGeo& q, int r, int k, int n) {
    if (k >= n) return -1;
    int dx, dy, dz;
    shell_offset(r, k, dx, dy, dz);
    const int x = q.bx + dx, y = q.by + dy, z = q.bz + dz;
    if (x < 0 || y < 0 || z < 0 || x >= s.bnx || y >= s.bny || z >= s.bnz) return -1;
    return s.brick_begin + (static_cast<int64_t>(z) * s.bny + y) * s.bnx + x;
}

// Upper bound on the distance from point c (corner-relative) to a large triangle:
// the distance to its nearest edge point (segments), plus rounding margin.
__device__ __forceinline__ float seg_dist(float px, float py, float pz, float ax, float ay, float az,
                                          float bx, float by, float bz) {
    float ex = bx - ax, ey = by - ay, ez = bz - az;
    float qx = px - ax, qy = py - ay, qz = pz - az;
    float ee = ex * ex + ey * ey + ez * ez;
    float t = ee > 0.f ? __saturatef((qx * ex + qy * ey + qz * ez) / ee) : 0.f;
    qx -= t * ex; qy -= t * ey; qz -= t * ez;
    return sqrtf(qx * qx + qy * qy + qz * qz);
}

__device__ __forceinline__ float large_upper(const double* __restrict__ soup, int64_t t,
                                             const double* K, float cx, float cy, float cz,
                                             float tol) {
    d3 a, b, c;
    load_soup(soup, t, a, b, c);
    float ax = static_cast<float>(a.x - K[0]), ay = static_cast<float>(a.y - K[1]),
          az = static_cast<float>(a.z - K[2]);
    float bx = static_cast<float>(b.x - K[0]), by = static_cast<float>(b.y - K[1]),
          bz = static_cast<float>(b.z - K[2]);
    float qx = static_cast<float>(c.x - K[0]), qy = static_cast<float>(c.y - K[1]),
          qz = static_cast<float>(c.z - K[2]);
    float d = fminf(seg_dist(cx, cy, cz, ax, ay, az, bx, by, bz),
                    fminf(seg_dist(cx, cy, cz, bx, by, bz, qx, qy, qz),
                          seg_dist(cx, cy, cz, qx, qy, qz, ax, ay, az)));
    return d * (1.f + 16.f * kU32) + tol;
}

__device__ __forceinline__ float aabb_dist(float cx, float cy, float cz, float4 lo, float4 hi) {
    float dx = fmaxf(0.f, fmaxf(lo.x - cx, cx - hi.x));
    float dy = fmaxf(0.f, fmaxf(lo.y - cy, cy - hi.y));
    float dz = fmaxf(0.f, fmaxf(lo.z - cz, cz - hi.z));
    return sqrtf(dx * dx + dy * dy + dz * dz) * (1.f - 8.f * kU32);
}

// The entries of a group of 32 bins (lane L holds bin L's range [b0, b1)) as one
// list, in bin order and then entry order: the order of a loop over the bins. The
// warp takes 32 x R entries per round (R loads in flight per lane, across bin
// boundaries); f(e, ok) gets the R entry positions of this lane and whether each
// exists. The trip count is warp-uniform, so f may use warp votes.
template <int kWalkRounds, class F>
__device__ __forceinline__ void for_group_entries(int64_t b0, int64_t b1, int lane, F&& f) {
    const int len = static_cast<int>(b1 - b0);
    int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    const int excl = inc - len;
    for (int base = 0; base < total; base += 32 * kWalkRounds) {
        int64_t e[kWalkRounds];
        bool ok[kWalkRounds];
#pragma unroll
        for (int j = 0; j < kWalkRounds; ++j) {
            const int v = base + 32 * j + lane;
            // owner bin: the number of bins whose inclusive end is <= v
            int lo = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xffffffffu, inc, lo + step - 1) <= v) lo += step;
            const int L = min(lo, 31);
            const int s0 = __shfl_sync(0xffffffffu, excl, L);
            const int64_t bb = __shfl_sync(0xffffffffu, b0, L);
            ok[j] = v < total;
            e[j] = bb + (v - s0);
        }
        f(e, ok);
    }
}

// Candidate lists, one kernel: per brick
//   1. an upper bound U on the distance from its centre to the surface, from the nearest
//      binned centroid (a point of the surface) and the large triangles' edges;
//   2. the count of the triangles that can be nearest to some cell of the brick: every
//      triangle whose lower bound |c - c_t| - e_t - r_B can be <= U + r_B, cut by the box test
//      around that centroid (a brick's sphere gives away 2 r_B in every direction, most of the
//      list of a brick far from the surface);
//   3. space for them (an atomic on the total; the lists' order in memory means nothing) and
//      the entries, if they fit.
// Bins are taken in Chebyshev shells around the brick; a bin's ball (k_bin_balls) is tested
// before its entries, which lie in order (bin_info). W warps per brick (8 / W bricks per
// CTA), by the mesh (MeshSeg::walk_warps): the walks of the bricks deep inside a closed
// surface, and of bricks with thousands of triangles each, set the kernel's time when the
// rest of the GPU has run dry. Each shell's 32-bin groups are split into contiguous ranges,
// one per warp, and each warp writes its own entries after those of the warps before it;
// the bound is reduced over the brick's warps after each shell (a named barrier per brick).
// (231x247x256 surface, 65k triangles, W = 4: 0.57 + 0.87 ms for a counting and a writing
// kernel that gathered every entry of every shell's bins -> 0.56 ms -> 0.52 ms in the order
// below.)
constexpr int kWalkThreads = 256;

// Brick number k of the mesh when they are taken from the middle of the grid outward, layer
// by layer and row by row: the lists of the bricks deep inside a closed surface are the
// longest, and a long one taken last would be waited for (231x247x256: 0.61 -> 0.52 ms; 24
// meshes, which are taken by triangles per brick besides: 2.20 -> 2.00 ms).
__device__ __forceinline__ int64_t centre_first(const MeshSeg& s, int64_t k) {
    auto outward = [](int i, int n) { return n / 2 + ((i & 1) ? -((i + 1) / 2) : i / 2); };
    const int x = static_cast<int>(k % s.bnx), y = static_cast<int>(k / s.bnx % s.bny),
              z = static_cast<int>(k / (static_cast<int64_t>(s.bnx) * s.bny));
    return (static_cast<int64_t>(outward(z, s.bnz)) * s.bny + outward(y, s.bny)) * s.bnx + outward(x, s.bnx);
}


template <int kWalkRounds>
__device__ __forceinline__ void brick_walk(const MeshSeg& turn, const MeshSeg* __restrict__ segs, int nseg,
           const double* __restrict__ soup, const float4* __restrict__ tinfo,
           const float4* __restrict__ tlo, const float4* __restrict__ thi,
           const int64_t* __restrict__ bin_off, const int* __restrict__ bin_list,
           const float4* __restrict__ bin_info, const float4* __restrict__ bin_ball,
           const float* __restrict__ bin_reach, const int* __restrict__ large_list,
           int* __restrict__ cand_cnt, int64_t* __restrict__ cand_rng, int* __restrict__ cand,
           float4* __restrict__ cand_c, int64_t cap, float* __restrict__ brick_emax,
           Stats* __restrict__ st, unsigned long long* __restrict__ queue) {
    constexpr int kWarps = kWalkThreads / 32;
    __shared__ float4 s_q[kWarps];
    __shared__ int s_c[kWarps];
    __shared__ long long s_off[kWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const MeshSeg& s = segs[turn.walk_seg];
    const int W = s.walk_warps;
    const int slot = wid / W, sub = wid % W;  // brick within the CTA, warp within the brick
    const int first = slot * W;               // the brick's first warp
    int64_t lb = (blockIdx.x - turn.walk_begin) * (kWarps / W) + slot;
    if (lb >= static_cast<int64_t>(s.bnx) * s.bny * s.bnz) return;  // uniform over the brick's warps
    lb = centre_first(s, lb);
    const int64_t gb = s.brick_begin + lb;
    auto brick_sync = [&]() {
        if (W == 1) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(32 * W) : "memory");
    };
    const BrickGeo q = brick_geo(s, lb);
    const float bw = static_cast<float>(s.brick * s.g.h);
    const float tol = list_tol(s.scale);
    const float emax = s.emax;
    // the last shell with a bin in the grid
    const int rmax = max(max(max(q.bx, s.bnx - 1 - q.bx), max(q.by, s.bny - 1 - q.by)), max(q.bz, s.bnz - 1 - q.bz));
    // the nearest centroid of the brick's warps (called by each of its threads, at points
    // uniform over the brick): p its offset and squared distance, id its triangle. Ties go to
    // the lowest triangle, so that the lists do not depend on the bins' order.
    auto brick_nearest = [&](float4& p, int& id) {
        const unsigned m = __reduce_min_sync(0xffffffffu, __float_as_uint(p.w));
        const int best = __reduce_min_sync(0xffffffffu, __float_as_uint(p.w) == m ? id : INT_MAX);
        const int src = __ffs(__ballot_sync(0xffffffffu, __float_as_uint(p.w) == m && id == best)) - 1;
        p.x = __shfl_sync(0xffffffffu, p.x, src);
        p.y = __shfl_sync(0xffffffffu, p.y, src);
        p.z = __shfl_sync(0xffffffffu, p.z, src);
        p.w = __uint_as_float(m);
        id = best;
        if (W == 1) return;
        if (lane == 0) {
            s_q[wid] = p;
            s_c[wid] = id;
        }
        brick_sync();
        for (int w = 0; w < W; ++w) {
            const float4 o = s_q[first + w];
            const int oid = s_c[first + w];
            if (o.w < p.w || (o.w == p.w && oid < id)) {
                p = o;
                id = oid;
            }
        }
        brick_sync();
    };
    // this warp's contiguous range [g0, g1) of the 32-bin groups of a shell of n bins
    auto range = [&](int n, int& g0, int& g1) {
        const int ng = (n + 31) / 32;
        g0 = static_cast<int>(static_cast<int64_t>(ng) * sub / W);
        g1 = static_cast<int>(static_cast<int64_t>(ng) * (sub + 1) / W);
    };
    // ---- 1. the bound. UL: from the large triangles; U: that or the nearest centroid's
    float UL = FLT_MAX;
    for (int64_t e = s.large_begin + 32 * sub + lane; e < s.large_end; e += 32 * W) {
        const int t = large_list[e];
        if (tlo[t].w == 0.f)  // (a thin triangle's distance may be none: it bounds nothing)
            UL = fminf(UL, large_upper(soup, t, s.g.corner, q.cx, q.cy, q.cz, tol));
    }
    {
        float4 p = make_float4(0.f, 0.f, 0.f, UL);
        int none = INT_MAX;
        brick_nearest(p, none);
        UL = p.w;
    }
    float4 near = make_float4(0.f, 0.f, 0.f, FLT_MAX);
    int near_t = INT_MAX;
    float U = UL;
    for (int r = 0; r <= rmax; ++r) {
        if (r > 0 && (r - 1) * bw > U) break;  // farther bins cannot lower U
        const int n = shell_count(r);
        int g0, g1;
        range(n, g0, g1);
        for (int g = g0; g < g1; ++g) {
            const int64_t bin = shell_bin(s, q, r, 32 * g + lane, n);
            int64_t b0 = 0, b1 = 0;
            if (bin >= 0) {
                const float4 ball = bin_ball[bin];
                const float dx = ball.x - q.cx, dy = ball.y - q.cy, dz = ball.z - q.cz;
                // only bins with a centroid that can be nearer than the nearest so far
                const float reach = fminf(U, sqrt_approx(near.w) * (1.f + 8.f * kU32)) + ball.w + tol;
                if (ball.w >= 0.f && !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > reach * reach * (1.f + 16.f * kU32))) {
                    b0 = bin_off[bin];
                    b1 = bin_off[bin + 1];
                }
            }
            for_group_entries<kWalkRounds>(b0, b1, lane, [&](const int64_t* e, const bool* ok) {
                float4 t[kWalkRounds];
#pragma unroll
                for (int j = 0; j < kWalkRounds; ++j)
                    t[j] = ok[j] ? bin_info[e[j]] : make_float4(FLT_MAX, 0.f, 0.f, 0.f);
#pragma unroll
                for (int j = 0; j < kWalkRounds; ++j) {
                    const float x = t[j].x - q.cx, y = t[j].y - q.cy, z = t[j].z - q.cz;
                    const float d2 = fmaf(x, x, fmaf(y, y, z * z));
                    if (d2 <= near.w && ok[j]) {
                        const int id = bin_list[e[j]];
                        if (d2 < near.w || id < near_t) {
                            near = make_float4(x, y, z, d2);
                            near_t = id;
                        }
                    }
                }
            });
        }
        brick_nearest(near, near_t);
        U = fminf(UL, near.w < FLT_MAX ? sqrtf(near.w) * (1.f + 8.f * kU32) + tol : FLT_MAX);
    }
    // ---- 2. candidates: lower bound <= U + 2 r_B (+ margins). The relative margin (4e-5,
    // about 670 u) covers four stated FP32 errors 48u (d + 2e + 2r) beyond any cell's
    // distance (e at most two bricks here; larger triangles are always considered): the
    // exact FP64 path's near-ties need them, the mixed path two
    const float lim = (U + 2.f * q.rb) * (1.f + 4e-5f) + 2.f * tol;
    const bool boxed = near.w < FLT_MAX;
    BoxTest box;
    if (boxed) {
        const float h = static_cast<float>(s.g.h);
        box = box_test(near.x, near.y, near.z, 0.5f * (q.x1 - q.x0 - 1) * h, 0.5f * (q.y1 - q.y0 - 1) * h,
                       0.5f * (q.z1 - q.z0 - 1) * h, q.rb, fmaf(4e-5f, U + 2.f * q.rb, 4.f * tol), tol);
    }
    const unsigned below = (1u << lane) - 1u;
    // whether a ball (a bin's or a triangle's, centre from the brick's centre) can matter
    auto reaches = [&](float x, float y, float z, float w) {
        const float d2 = fmaf(x, x, fmaf(y, y, z * z)), l = lim + w;  // |v - c| - w >= d - r_B - w
        return !(d2 > l * l * (1.f + 16.f * kU32)) && (!boxed || box_ball(box, x, y, z, w, tol));
    };
    // walks this warp's groups of every shell; f(take, entry, info) per kWalkRounds entries of
    // each lane, in walk order, called by the whole warp
    auto walk = [&](auto&& f) {
        for (int r = 0; r <= rmax; ++r) {
            if (r > 0 && (r - 1) * bw - emax > lim) break;
            const int n = shell_count(r);
            int g0, g1;
            range(n, g0, g1);
            for (int g = g0; g < g1; ++g) {
                const int64_t bin = shell_bin(s, q, r, 32 * g + lane, n);
                int64_t b0 = 0, b1 = 0;
                if (bin >= 0) {
                    const float4 ball = bin_ball[bin];
                    if (ball.w >= 0.f && reaches(ball.x - q.cx, ball.y - q.cy, ball.z - q.cz, bin_reach[bin])) {
                        b0 = bin_off[bin];
                        b1 = bin_off[bin + 1];
                    }
                }
                for_group_entries<kWalkRounds>(b0, b1, lane, [&](const int64_t* e, const bool* ok) {
                    float4 t[kWalkRounds];
#pragma unroll
                    for (int j = 0; j < kWalkRounds; ++j)
                        t[j] = ok[j] ? bin_info[e[j]] : make_float4(0.f, 0.f, 0.f, 0.f);
                    bool take[kWalkRounds];
#pragma unroll
                    for (int j = 0; j < kWalkRounds; ++j)
                        take[j] = ok[j] && reaches(t[j].x - q.cx, t[j].y - q.cy, t[j].z - q.cz, t[j].w);
                    f(take, e, t);
                });
            }
        }
    };
    // the always-considered large triangles, by the brick's first warp
    auto walk_large = [&](auto&& f) {
        for (int64_t e0 = s.large_begin; e0 < s.large_end; e0 += 32) {
            const int64_t e = e0 + lane;
            bool take = false;
            int t = 0;
            float4 ti = make_float4(0.f, 0.f, 0.f, 0.f);
            if (e < s.large_end) {
                t = large_list[e];
                take = aabb_dist(q.cx, q.cy, q.cz, tlo[t], thi[t]) <= lim;  // d(v,t) >= d - r_B must reach U + r_B
                ti = tinfo[t];
            }
            f(take, t, ti);
        }
    };
    int mine = 0;
    auto count = [&](bool take) { mine += __popc(__ballot_sync(0xffffffffu, take)); };
    if (sub == 0) walk_large([&](bool take, int, const float4&) { count(take); });
    walk([&](const bool* take, const int64_t*, const float4*) {
#pragma unroll
        for (int j = 0; j < kWalkRounds; ++j) count(take[j]);
    });
    // ---- 3. the list's place, and the entries
    if (lane == 0) s_c[wid] = mine;
    brick_sync();
    int before = 0, total = 0;
    for (int w = 0; w < W; ++w) {
        if (w < sub) before += s_c[first + w];
        total += s_c[first + w];
    }
    if (sub == 0 && lane == 0) {
        const long long at = static_cast<long long>(atomicAdd(&st->candidates, static_cast<unsigned long long>(total)));
        s_off[first] = at;
        cand_cnt[gb] = total;
        const bool fits = at + total <= cap;
        cand_rng[2 * gb] = fits ? at : 0;
        cand_rng[2 * gb + 1] = fits ? at + total : 0;
    }
    brick_sync();
    int64_t at = s_off[first];
    if (at + total > cap) {  // uniform over the brick: the lists are sized and walked again
        if (sub == 0 && lane == 0) atomicMax(queue, kQueueClosed);
        return;
    }
    at += before;
    float bemax = 0.f;
    // a list entry: the triangle and, for the warp-per-sub-brick evaluation, its centroid from
    // the brick's centre and its radius, so that the scans read them in order (each brick's
    // list is scanned twice by its 64 sub-bricks)
    auto put = [&](bool take, int t, const float4& ti) {
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) {
            const int64_t k = at + __popc(m & below);
            cand[k] = t;
            if (cand_c) cand_c[k] = make_float4(ti.x - q.cx, ti.y - q.cy, ti.z - q.cz, ti.w);
            bemax = fmaxf(bemax, ti.w);
        }
        at += __popc(m);
    };
    if (sub == 0) walk_large(put);
    walk([&](const bool* take, const int64_t* e, const float4* ti) {
        int id[kWalkRounds];  // (loaded together)
#pragma unroll
        for (int j = 0; j < kWalkRounds; ++j) id[j] = take[j] ? bin_list[e[j]] : 0;
#pragma unroll
        for (int j = 0; j < kWalkRounds; ++j) put(take[j], id[j], ti[j]);
    });
    {
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        bemax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(bemax)));
        if (W > 1) {
            p.w = bemax;
            if (lane == 0) s_q[wid] = p;
            brick_sync();
            for (int w = 0; w < W; ++w) bemax = fmaxf(bemax, s_q[first + w].w);
        }
        if (sub == 0 && lane == 0) brick_emax[gb] = bemax;
    }
}

// Eight-warp bricks have long walks of full groups and take eight entries per lane and round,
// the others four; a launch with eight-warp bricks has 122 registers and two CTAs per SM, one
// without 80 and three, which leaves room for the occupancy passes beside it. (137^3 around
// 128k triangles 0.43 -> 0.36 ms, 118x126x130 around 65k 0.40 -> 0.32, 24 meshes 1.98 ->
// 1.68 with eight; 231x247x256, four warps: 0.46 alone with two CTAs against 0.52 with three,
// but the whole call 0.4 % slower.)
template <bool EIGHT>
__global__ void __launch_bounds__(kWalkThreads, EIGHT ? 2 : 3)
k_brick_walk(const MeshSeg* __restrict__ segs, int nseg,
             const double* __restrict__ soup, const float4* __restrict__ tinfo,
             const float4* __restrict__ tlo, const float4* __restrict__ thi,
             const int64_t* __restrict__ bin_off, const int* __restrict__ bin_list,
             const float4* __restrict__ bin_info, const float4* __restrict__ bin_ball,
             const float* __restrict__ bin_reach, const int* __restrict__ large_list,
             int* __restrict__ cand_cnt, int64_t* __restrict__ cand_rng, int* __restrict__ cand,
             float4* __restrict__ cand_c, int64_t cap, float* __restrict__ brick_emax,
             Stats* __restrict__ st, unsigned long long* __restrict__ queue) {
    const MeshSeg& turn = segs[find_seg<&MeshSeg::walk_begin>(segs, nseg, blockIdx.x)];
    if (EIGHT && segs[turn.walk_seg].walk_warps == 8)
        brick_walk<8>(turn, segs, nseg, soup, tinfo, tlo, thi, bin_off, bin_list, bin_info, bin_ball, bin_reach, large_list, cand_cnt, cand_rng, cand, cand_c, cap, brick_emax, st, queue);
    else
        brick_walk<4>(turn, segs, nseg, soup, tinfo, tlo, thi, bin_off, bin_list, bin_info, bin_ball, bin_reach, large_list, cand_cnt, cand_rng, cand, cand_c, cap, brick_emax, st, queue);
}

// ------------------------------------------------------------------ evaluation
constexpr int kChunk = 64;  // candidates staged per round

// Cell owned by (thread, slot) inside a brick of edge B.
template <int B, int THREADS>
struct CellMap {
    static constexpr int VPT = B * B * B / THREADS;
    __device__ static void cell(int tid, int v, int& x, int& y, int& z) {
        // threads tile x (fastest), then y, then z-slabs; each thread owns VPT cells in z
        x = tid % B;
        y = (tid / B) % B;
        int zslab = tid / (B * B);
        z = zslab * VPT + v;
    }
};

// Plain FP64: CTA per brick (persistent over a work list), THREADS threads.
template <int B, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_sdf_fp64(const MeshSeg* __restrict__ segs, int nseg, const uint32_t* __restrict__ work,
           int64_t nwork, unsigned long long* __restrict__ queue, const double* __restrict__ soup,
           const float4* __restrict__ tinfo, const int64_t* __restrict__ cand_rng,
           const int* __restrict__ cand, Out o, Stats* __restrict__ st) {
    using M = CellMap<B, THREADS>;
    constexpr int VPT = M::VPT;
    __shared__ double sv[kChunk][12];  // a, b, c, centroid (FP64)
    __shared__ double srad[kChunk];
    __shared__ int sid[kChunk];
    __shared__ int64_t s_item;
    const int tid = threadIdx.x;
    unsigned long long evals = 0;
    for (;;) {
        if (tid == 0) s_item = static_cast<int64_t>(atomicAdd(queue, 1ull));
        __syncthreads();
        const int64_t item = s_item;
        __syncthreads();
        if (item >= nwork) break;
        const int64_t gb = static_cast<int64_t>(work[item]);
        const int si = find_seg<&MeshSeg::brick_begin>(segs, nseg, gb);
        const MeshSeg& s = segs[si];
        const BrickGeo q = brick_geo(s, gb - s.brick_begin);
        const GridDesc g = s.g;
        d3 p[VPT];
        bool valid[VPT];
        double best[VPT], bestd[VPT];
        int bt[VPT], br[VPT];
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            int x, y, z;
            M::cell(tid, v, x, y, z);
            x += q.x0; y += q.y0; z += q.z0;
            valid[v] = x < q.x1 && y < q.y1 && z < q.z1;
            p[v] = {cell_center(g.corner[0], x, g.h), cell_center(g.corner[1], y, g.h),
                    cell_center(g.corner[2], z, g.h)};
            best[v] = DBL_MAX;
            bestd[v] = DBL_MAX;
            bt[v] = INT_MAX;
            br[v] = 0;
        }
        const int64_t c0 = cand_rng[2 * gb], c1 = cand_rng[2 * gb + 1];
        for (int64_t base = c0; base < c1; base += kChunk) {
            const int n = static_cast<int>(c1 - base < kChunk ? c1 - base : kChunk);
            __syncthreads();
            for (int k = tid; k < n; k += THREADS) {
                int t = cand[base + k];
                d3 a, b, c;
                load_soup(soup, t, a, b, c);
                sv[k][0] = a.x; sv[k][1] = a.y; sv[k][2] = a.z;
                sv[k][3] = b.x; sv[k][4] = b.y; sv[k][5] = b.z;
                sv[k][6] = c.x; sv[k][7] = c.y; sv[k][8] = c.z;
                float4 ti = tinfo[t];
                sv[k][9] = g.corner[0] + ti.x;
                sv[k][10] = g.corner[1] + ti.y;
                sv[k][11] = g.corner[2] + ti.z;
                srad[k] = static_cast<double>(ti.w) * (1.0 + 1e-6) + 1e-9 * s.scale;
                sid[k] = t;
            }
            __syncthreads();
            for (int k = 0; k < n; ++k) {
                // warp-uniform skip: the bounding sphere is beyond every lane's best
                bool need = false;
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    double dx = p[v].x - sv[k][9], dy = p[v].y - sv[k][10], dz = p[v].z - sv[k][11];
                    double lim = bestd[v] + srad[k];
                    need |= valid[v] && (bestd[v] == DBL_MAX || dx * dx + dy * dy + dz * dz <= lim * lim);
                }
                if (!__any_sync(0xffffffffu, need)) continue;
                const d3 a{sv[k][0], sv[k][1], sv[k][2]}, b{sv[k][3], sv[k][4], sv[k][5]},
                    c{sv[k][6], sv[k][7], sv[k][8]};
                const int t = sid[k];
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    if (!valid[v]) continue;
                    int reg;
                    double d2 = ericson(p[v], a, b, c, &reg);
                    ++evals;
                    if (d2 < best[v] || (d2 == best[v] && t < bt[v])) {
                        best[v] = d2;
                        bt[v] = t;
                        br[v] = reg;
                        bestd[v] = sqrt(d2) * (1.0 + 1e-9);
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            if (!valid[v]) continue;
            int x, y, z;
            M::cell(tid, v, x, y, z);
            x += q.x0; y += q.y0; z += q.z0;
            int64_t idx = s.vox_begin + (static_cast<int64_t>(z) * g.ny + y) * g.nx + x;
            write_cell(o, idx, __dsqrt_rn(best[v]), bt[v], br[v]);
        }
    }
    long long ev = warp_sum(static_cast<long long>(evals));
    if ((tid & 31) == 0 && ev) {
        atomicAdd(&st->evaluations, static_cast<unsigned long long>(ev));
        atomicAdd(&st->fp64_evaluations, static_cast<unsigned long long>(ev));
    }
}

// FP32 record of a candidate, recentred on the brick centre.
struct alignas(16) Rec32 {
    float v0[3], v1[3], v2[3];   // vertices
    float e0[3], e1[3], e2[3];   // edges v1-v0, v2-v1, v0-v2
    float nn[3];                 // unit normal (from FP64)
    float m0[3], m1[3], m2[3];   // in-plane inward edge normals
    float inv[3];                // 1 / |e_k|^2 (0 for a degenerate edge)
    float cen[3], rad;           // bounding sphere
    float ok;                    // 1: plane branch allowed (non-degenerate)
    int tid;
    float pad_[1];
};
static_assert(sizeof(Rec32) == 160, "record layout");

__device__ __forceinline__ void make_rec(Rec32& r, const d3& a, const d3& b, const d3& c,
                                         const double* cb, float rad, int t) {
    float v[9] = {static_cast<float>(a.x - cb[0]), static_cast<float>(a.y - cb[1]),
                  static_cast<float>(a.z - cb[2]), static_cast<float>(b.x - cb[0]),
                  static_cast<float>(b.y - cb[1]), static_cast<float>(b.z - cb[2]),
                  static_cast<float>(c.x - cb[0]), static_cast<float>(c.y - cb[1]),
                  static_cast<float>(c.z - cb[2])};
    for (int k = 0; k < 3; ++k) {
        r.v0[k] = v[k]; r.v1[k] = v[3 + k]; r.v2[k] = v[6 + k];
        r.e0[k] = v[3 + k] - v[k];
        r.e1[k] = v[6 + k] - v[3 + k];
        r.e2[k] = v[k] - v[6 + k];
    }
    // normal in FP64 from the FP64 vertices, then normalised in FP32
    double ux = b.x - a.x, uy = b.y - a.y, uz = b.z - a.z;
    double wx = c.x - a.x, wy = c.y - a.y, wz = c.z - a.z;
    double nx = uy * wz - uz * wy, ny = uz * wx - ux * wz, nz = ux * wy - uy * wx;
    double nl = sqrt(nx * nx + ny * ny + nz * nz);
    float ok = nl > 0.0 ? 1.f : 0.f;
    float n3[3] = {0.f, 0.f, 0.f};
    if (nl > 0.0) {
        n3[0] = static_cast<float>(nx / nl);
        n3[1] = static_cast<float>(ny / nl);
        n3[2] = static_cast<float>(nz / nl);
    }
    r.nn[0] = n3[0]; r.nn[1] = n3[1]; r.nn[2] = n3[2];
    const float* E[3] = {r.e0, r.e1, r.e2};
    float* Mv[3] = {r.m0, r.m1, r.m2};
    for (int k = 0; k < 3; ++k) {
        const float* e = E[k];
        // n x e points into the triangle for a counter-clockwise (about n) edge
        Mv[k][0] = n3[1] * e[2] - n3[2] * e[1];
        Mv[k][1] = n3[2] * e[0] - n3[0] * e[2];
        Mv[k][2] = n3[0] * e[1] - n3[1] * e[0];
        float ee = e[0] * e[0] + e[1] * e[1] + e[2] * e[2];
        r.inv[k] = ee > 0.f ? 1.f / ee : 0.f;
    }
    r.cen[0] = (v[0] + v[3] + v[6]) * (1.f / 3.f);
    r.cen[1] = (v[1] + v[4] + v[7]) * (1.f / 3.f);
    r.cen[2] = (v[2] + v[5] + v[8]) * (1.f / 3.f);
    r.rad = rad * (1.f + 64.f * kU32);
    r.ok = ok;
    r.tid = t;
}

// FP32 squared distance from p to the recorded triangle; region in Ericson's
// numbering (0 a, 1 b, 2 ab, 3 c, 4 ac, 5 bc, 6 interior).
__device__ __forceinline__ float dist32(const Rec32& r, float px, float py, float pz, int* reg) {
    float pax = px - r.v0[0], pay = py - r.v0[1], paz = pz - r.v0[2];
    float pbx = px - r.v1[0], pby = py - r.v1[1], pbz = pz - r.v1[2];
    float pcx = px - r.v2[0], pcy = py - r.v2[1], pcz = pz - r.v2[2];
    float s0 = r.m0[0] * pax + r.m0[1] * pay + r.m0[2] * paz;
    float s1 = r.m1[0] * pbx + r.m1[1] * pby + r.m1[2] * pbz;
    float s2 = r.m2[0] * pcx + r.m2[1] * pcy + r.m2[2] * pcz;
    if (r.ok > 0.f && s0 >= 0.f && s1 >= 0.f && s2 >= 0.f) {
        float dp = r.nn[0] * pax + r.nn[1] * pay + r.nn[2] * paz;
        *reg = 6;
        return dp * dp;
    }
    float t0 = __saturatef((pax * r.e0[0] + pay * r.e0[1] + paz * r.e0[2]) * r.inv[0]);
    float qx = pax - t0 * r.e0[0], qy = pay - t0 * r.e0[1], qz = paz - t0 * r.e0[2];
    float d0 = qx * qx + qy * qy + qz * qz;
    float t1 = __saturatef((pbx * r.e1[0] + pby * r.e1[1] + pbz * r.e1[2]) * r.inv[1]);
    qx = pbx - t1 * r.e1[0]; qy = pby - t1 * r.e1[1]; qz = pbz - t1 * r.e1[2];
    float d1 = qx * qx + qy * qy + qz * qz;
    float t2 = __saturatef((pcx * r.e2[0] + pcy * r.e2[1] + pcz * r.e2[2]) * r.inv[2]);
    qx = pcx - t2 * r.e2[0]; qy = pcy - t2 * r.e2[1]; qz = pcz - t2 * r.e2[2];
    float d2 = qx * qx + qy * qy + qz * qz;
    float d = d0;
    int g = t0 <= 0.f ? 0 : (t0 >= 1.f ? 1 : 2);
    if (d1 < d) { d = d1; g = t1 <= 0.f ? 1 : (t1 >= 1.f ? 3 : 5); }
    if (d2 < d) { d = d2; g = t2 <= 0.f ? 3 : (t2 >= 1.f ? 0 : 4); }
    *reg = g;
    return d;
}

template <int B, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_sdf_mixed(const MeshSeg* __restrict__ segs, int nseg, const uint32_t* __restrict__ work,
            int64_t nwork, unsigned long long* __restrict__ queue, const double* __restrict__ soup,
            const float4* __restrict__ tinfo, const int64_t* __restrict__ cand_rng,
            const int* __restrict__ cand, const float* __restrict__ brick_emax, float band_cells,
            Out o, Stats* __restrict__ st) {
    using M = CellMap<B, THREADS>;
    constexpr int VPT = M::VPT;
    __shared__ Rec32 rec[kChunk];
    __shared__ int64_t s_item;
    __shared__ int s_band;
    const int tid = threadIdx.x;
    unsigned long long evals = 0, evals64 = 0, bandc = 0;
    for (;;) {
        if (tid == 0) {
            s_item = static_cast<int64_t>(atomicAdd(queue, 1ull));
            s_band = 0;
        }
        __syncthreads();
        const int64_t item = s_item;
        if (item >= nwork) break;
        const int64_t gb = static_cast<int64_t>(work[item]);
        const int si = find_seg<&MeshSeg::brick_begin>(segs, nseg, gb);
        const MeshSeg& s = segs[si];
        const BrickGeo q = brick_geo(s, gb - s.brick_begin);
        const GridDesc g = s.g;
        // brick centre in FP64 (the recentring origin)
        const double cb[3] = {g.corner[0] + 0.5 * (q.x0 + q.x1) * g.h,
                              g.corner[1] + 0.5 * (q.y0 + q.y1) * g.h,
                              g.corner[2] + 0.5 * (q.z0 + q.z1) * g.h};
        float px[VPT], py[VPT], pz[VPT], best[VPT], bestd[VPT];
        int bt[VPT], br[VPT];
        bool valid[VPT];
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            int x, y, z;
            M::cell(tid, v, x, y, z);
            x += q.x0; y += q.y0; z += q.z0;
            valid[v] = x < q.x1 && y < q.y1 && z < q.z1;
            px[v] = static_cast<float>(cell_center(g.corner[0], x, g.h) - cb[0]);
            py[v] = static_cast<float>(cell_center(g.corner[1], y, g.h) - cb[1]);
            pz[v] = static_cast<float>(cell_center(g.corner[2], z, g.h) - cb[2]);
            best[v] = FLT_MAX;
            bestd[v] = FLT_MAX;
            bt[v] = INT_MAX;
            br[v] = 0;
        }
        const int64_t c0 = cand_rng[2 * gb], c1 = cand_rng[2 * gb + 1];
        for (int64_t base = c0; base < c1; base += kChunk) {
            const int n = static_cast<int>(c1 - base < kChunk ? c1 - base : kChunk);
            __syncthreads();
            for (int k = tid; k < n; k += THREADS) {
                int t = cand[base + k];
                d3 a, b, c;
                load_soup(soup, t, a, b, c);
                make_rec(rec[k], a, b, c, cb, tinfo[t].w, t);
            }
            __syncthreads();
            for (int k = 0; k < n; ++k) {
                const Rec32& r = rec[k];
                bool need = false;
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    float dx = px[v] - r.cen[0], dy = py[v] - r.cen[1], dz = pz[v] - r.cen[2];
                    float lim = bestd[v] + r.rad;
                    need |= valid[v] && dx * dx + dy * dy + dz * dz <= lim * lim;
                }
                if (!__any_sync(0xffffffffu, need)) continue;
#pragma unroll
                for (int v = 0; v < VPT; ++v) {
                    if (!valid[v]) continue;
                    int reg;
                    float d2 = dist32(r, px[v], py[v], pz[v], &reg);
                    ++evals;
                    if (d2 < best[v] || (d2 == best[v] && r.tid < bt[v])) {
                        best[v] = d2;
                        bt[v] = r.tid;
                        br[v] = reg;
                        bestd[v] = sqrtf(d2) * (1.f + 4.f * kU32) + 1e-30f;
                    }
                }
            }
        }
        // stated FP32 error bound per cell and the FP64 band
        const float emx = brick_emax[gb];
        const float bandw = band_cells * static_cast<float>(g.h);
        float eb[VPT];
        bool inband[VPT];
        bool any_band = false;
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            float d = sqrtf(best[v]);
            eb[v] = 48.f * kU32 * (d + 2.f * emx + 2.f * q.rb) + 1e-30f;
            inband[v] = valid[v] && d <= bandw + eb[v];
            any_band |= inband[v];
        }
        if (any_band) s_band = 1;
        __syncthreads();
        double best64[VPT];
        int bt64[VPT], br64[VPT];
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            best64[v] = DBL_MAX;
            bt64[v] = INT_MAX;
            br64[v] = 0;
        }
        if (s_band) {
            // FP64 refinement over candidates within 2*eb of the FP32 best
            for (int64_t base = c0; base < c1; base += kChunk) {
                const int n = static_cast<int>(c1 - base < kChunk ? c1 - base : kChunk);
                __syncthreads();
                for (int k = tid; k < n; k += THREADS) {
                    int t = cand[base + k];
                    d3 a, b, c;
                    load_soup(soup, t, a, b, c);
                    make_rec(rec[k], a, b, c, cb, tinfo[t].w, t);
                }
                __syncthreads();
                for (int k = 0; k < n; ++k) {
                    const Rec32& r = rec[k];
#pragma unroll
                    for (int v = 0; v < VPT; ++v) {
                        if (!inband[v]) continue;
                        int reg;
                        float d2 = dist32(r, px[v], py[v], pz[v], &reg);
                        float lim = sqrtf(best[v]) + 2.f * eb[v];
                        if (sqrtf(d2) > lim * (1.f + 1e-6f)) continue;
                        d3 a, b, c;
                        load_soup(soup, r.tid, a, b, c);
                        int x, y, z;
                        M::cell(tid, v, x, y, z);
                        x += q.x0; y += q.y0; z += q.z0;
                        const d3 P{cell_center(g.corner[0], x, g.h), cell_center(g.corner[1], y, g.h),
                                   cell_center(g.corner[2], z, g.h)};
                        int r64;
                        double e2 = ericson(P, a, b, c, &r64);
                        ++evals64;
                        if (e2 < best64[v] || (e2 == best64[v] && r.tid < bt64[v])) {
                            best64[v] = e2;
                            bt64[v] = r.tid;
                            br64[v] = r64;
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int v = 0; v < VPT; ++v) {
            if (!valid[v]) continue;
            int x, y, z;
            M::cell(tid, v, x, y, z);
            x += q.x0; y += q.y0; z += q.z0;
            int64_t idx = s.vox_begin + (static_cast<int64_t>(z) * g.ny + y) * g.nx + x;
            if (inband[v]) {
                ++bandc;
                write_cell(o, idx, __dsqrt_rn(best64[v]), bt64[v], br64[v]);
                if (o.errbound) o.errbound[idx] = 0.f;
            } else {
                write_cell(o, idx, static_cast<double>(sqrtf(best[v])), bt[v], br[v]);
                if (o.errbound) o.errbound[idx] = eb[v];
            }
        }
        __syncthreads();
    }
    long long ev = warp_sum(static_cast<long long>(evals));
    long long ev64 = warp_sum(static_cast<long long>(evals64));
    long long bc = warp_sum(static_cast<long long>(bandc));
    if ((tid & 31) == 0) {
        if (ev) atomicAdd(&st->evaluations, static_cast<unsigned long long>(ev));
        if (ev64) atomicAdd(&st->fp64_evaluations, static_cast<unsigned long long>(ev64));
        if (bc) atomicAdd(&st->band_voxels, static_cast<unsigned long long>(bc));
    }
}

// Work model: per cell, K(v) = #{t : |p - c_t| - e_t <= |sdf(v)|}, the triangles
// whose bounding sphere reaches the distance sphere of the cell -- the minimal
// candidate set of any bounding-sphere-pruned exact search. out[0] = sum K over
// all cells, out[1] = sum K over cells with |sdf| <= band, out[2] = those cells.
template <int B, int THREADS>
__global__ void __launch_bounds__(THREADS)
k_count_K(const MeshSeg* __restrict__ segs, int nseg, int64_t nbricks,
          const float4* __restrict__ tinfo, const int64_t* __restrict__ cand_rng,
          const int* __restrict__ cand, const double* __restrict__ sdf64,
          const float* __restrict__ sdf32, float band_cells, unsigned long long* __restrict__ out) {
    using M = CellMap<B, THREADS>;
    constexpr int VPT = M::VPT;
    const int64_t gb = blockIdx.x;
    if (gb >= nbricks) return;
    const int si = find_seg<&MeshSeg::brick_begin>(segs, nseg, gb);
    const MeshSeg& s = segs[si];
    const BrickGeo q = brick_geo(s, gb - s.brick_begin);
    const GridDesc g = s.g;
    const float h = static_cast<float>(g.h);
    unsigned long long k_all = 0, k_band = 0, n_band = 0;
    for (int v = 0; v < VPT; ++v) {
        int x, y, z;
        M::cell(threadIdx.x, v, x, y, z);
        x += q.x0; y += q.y0; z += q.z0;
        if (!(x < q.x1 && y < q.y1 && z < q.z1 && z >= g.z0 && z < g.z1)) continue;
        int64_t idx = s.vox_begin + (static_cast<int64_t>(z - g.z0) * g.ny + y) * g.nx + x;
        float d = sdf64 ? static_cast<float>(fabs(sdf64[idx])) : fabsf(sdf32[idx]);
        float px = (x + 0.5f) * h, py = (y + 0.5f) * h, pz = (z + 0.5f) * h;
        unsigned kk = 0;
        for (int64_t e = cand_rng[2 * gb]; e < cand_rng[2 * gb + 1]; ++e) {
            float4 ti = tinfo[cand[e]];
            float dx = px - ti.x, dy = py - ti.y, dz = pz - ti.z;
            kk += sqrtf(dx * dx + dy * dy + dz * dz) - ti.w <= d;
        }
        kk = max(kk, 1u);
        k_all += kk;
        if (d <= band_cells * h) {
            k_band += kk;
            ++n_band;
        }
    }
    long long a = warp_sum(static_cast<long long>(k_all));
    long long b = warp_sum(static_cast<long long>(k_band));
    long long c = warp_sum(static_cast<long long>(n_band));
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(&out[0], static_cast<unsigned long long>(a));
        if (b) atomicAdd(&out[1], static_cast<unsigned long long>(b));
        if (c) atomicAdd(&out[2], static_cast<unsigned long long>(c));
    }
}

}  // namespace

// ------------------------------------------------------------------ launchers
void launch_sdf_tri_prep(const MeshSeg* segs, int nseg, int64_t ntris, const double* pts, const int* tris,
                         float4* tinfo, float4* tinfo_lo, void* trec, float4* tnorm, float4* tlo,
                         float4* thi,
                         int64_t* tbin, int* bincnt, int* large_cnt, unsigned* emax_bits, Stats* stats,
                         cudaStream_t st) {
    if (ntris == 0) return;
    k_sdf_tri_prep<<<static_cast<unsigned>((ntris + 255) / 256), 256, 0, st>>>(
        segs, nseg, ntris, pts, tris, tinfo, tinfo_lo, static_cast<TriRec*>(trec), tnorm, tlo, thi, tbin,
        bincnt, large_cnt, emax_bits, stats);
    CMG_LAUNCH();
}

void launch_bin_fill(int64_t ntris, const int64_t* tbin, const int64_t* bin_off, int* bincur,
                     const float4* tinfo, int* bin_list, float4* bin_info, int64_t nbins,
                     float4* bin_ball, float* bin_reach, const MeshSeg* segs, int nseg, int* large_cur,
                     int* large_list, cudaStream_t st) {
    if (ntris == 0) return;
    k_bin_fill<<<static_cast<unsigned>((ntris + 255) / 256), 256, 0, st>>>(
        ntris, tbin, bin_off, bincur, tinfo, bin_list, bin_info, segs, nseg, large_cur, large_list);
    CMG_LAUNCH();
    k_bin_balls<<<static_cast<unsigned>((nbins + 3) / 4), 128, 0, st>>>(nbins, bin_off, bin_info, segs, nseg,
                                                                        bin_ball, bin_reach);
    CMG_LAUNCH();
}

void launch_seg_finish(MeshSeg* segs, int nseg, const int* large_cnt, const unsigned* emax_bits,
                       cudaStream_t st) {
    k_seg_finish<<<1, kSegThreads, 0, st>>>(segs, nseg, large_cnt, emax_bits);
    CMG_LAUNCH();
}

int brick_walk_warps(int64_t nbricks, int64_t mesh_bricks, int64_t mesh_tris, int walk_warps) {
    if (walk_warps == 1 || walk_warps == 2 || walk_warps == 4) return walk_warps;
    // 8 while the bricks are few, or for a mesh whose bricks see hundreds of triangles each;
    // else 4 while 4-warp bricks fit about twice in the GPU, 2 up to twice that, then 1
    const int64_t sms = device_sms();
    if (nbricks <= 8 * sms || mesh_tris > 128 * mesh_bricks) return 8;
    return nbricks <= 32 * sms ? 4 : (nbricks <= 64 * sms ? 2 : 1);
}
int64_t brick_walk_ctas(int64_t mesh_bricks, int warps) {
    const int64_t per = kWalkThreads / 32 / warps;
    return (mesh_bricks + per - 1) / per;
}

void launch_brick_walk(const MeshSeg* segs, int nseg, int64_t ctas, const double* soup,
                       const float4* tinfo, const float4* tlo, const float4* thi,
                       const int64_t* bin_off, const int* bin_list, const float4* bin_info,
                       const float4* bin_ball, const float* bin_reach, const int* large_list,
                       int* cand_cnt, int64_t* cand_rng, int* cand, float4* cand_c, int64_t cap,
                       float* brick_emax, Stats* stats, unsigned long long* queue, bool eight,
                       cudaStream_t st) {
    if (ctas == 0) return;
    auto go = [&](auto kernel) {
        kernel<<<static_cast<unsigned>(ctas), kWalkThreads, 0, st>>>(
            segs, nseg, soup, tinfo, tlo, thi, bin_off, bin_list, bin_info, bin_ball, bin_reach, large_list,
            cand_cnt, cand_rng, cand, cand_c, cap, brick_emax, stats, queue);
    };
    if (eight) go(k_brick_walk<true>);
    else go(k_brick_walk<false>);
    CMG_LAUNCH();
}

void launch_count_K(int brick, const MeshSeg* segs, int nseg, int64_t nbricks, const float4* tinfo,
                    const int64_t* cand_rng, const int* cand, const double* sdf64,
                    const float* sdf32, float band_cells, unsigned long long* out,
                    cudaStream_t st) {
    if (nbricks == 0) return;
    if (brick == 4)
        k_count_K<4, 64><<<static_cast<unsigned>(nbricks), 64, 0, st>>>(
            segs, nseg, nbricks, tinfo, cand_rng, cand, sdf64, sdf32, band_cells, out);
    else if (brick == 16)
        k_count_K<16, 256><<<static_cast<unsigned>(nbricks), 256, 0, st>>>(
            segs, nseg, nbricks, tinfo, cand_rng, cand, sdf64, sdf32, band_cells, out);
    else
        k_count_K<8, 128><<<static_cast<unsigned>(nbricks), 128, 0, st>>>(
            segs, nseg, nbricks, tinfo, cand_rng, cand, sdf64, sdf32, band_cells, out);
    CMG_LAUNCH();
}

void launch_sdf_eval(int precision, int brick, const MeshSeg* segs, int nseg, const uint32_t* work,
                     int64_t nwork, unsigned long long* queue, const double* soup,
                     const float4* tinfo, const int64_t* cand_rng, const int* cand,
                     const float* brick_emax, float band_cells, const uint8_t* occ, float* sdf32,
                     double* sdf64, int* near_tri, uint8_t* near_reg, float* errbound, Stats* stats,
                     int grid, cudaStream_t st) {
    if (nwork == 0) return;
    Out o{occ, sdf32, sdf64, near_tri, near_reg, errbound};
    if (precision == kPrecMixed) {
        if (brick == 4)
            k_sdf_mixed<4, 64><<<grid, 64, 0, st>>>(segs, nseg, work, nwork, queue, soup, tinfo,
                                                    cand_rng, cand, brick_emax, band_cells, o, stats);
        else
            k_sdf_mixed<8, 128><<<grid, 128, 0, st>>>(segs, nseg, work, nwork, queue, soup, tinfo,
                                                      cand_rng, cand, brick_emax, band_cells, o,
                                                      stats);
    } else {
        if (brick == 4)
            k_sdf_fp64<4, 64><<<grid, 64, 0, st>>>(segs, nseg, work, nwork, queue, soup, tinfo,
                                                   cand_rng, cand, o, stats);
        else
            k_sdf_fp64<8, 128><<<grid, 128, 0, st>>>(segs, nseg, work, nwork, queue, soup, tinfo,
                                                     cand_rng, cand, o, stats);
    }
    CMG_LAUNCH();
}

}  // namespace cmg::gpu
