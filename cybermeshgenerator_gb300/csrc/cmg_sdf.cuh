// cmg_sdf.cuh — device pieces shared by the signed-distance kernels.
#pragma once

#include <cfloat>
#include <climits>

#include "cmg_device.cuh"
#include "cmg_types.h"

namespace cmg::gpu {
namespace sdf {

constexpr float kU32 = 5.9604645e-8f;  // 2^-24
constexpr double kU64 = 1.1102230246251565e-16;  // 2^-53

// ------------------------------------------------------------------ FP64 Ericson
// Squared distance and region, reference operation order (src/voxelize/
// voxelize.cpp:202-247); regions 0 a, 1 b, 2 ab, 3 c, 4 ac, 5 bc, 6 interior.
__device__ __forceinline__ double dot3r(double ax, double ay, double az, double bx, double by,
                                        double bz) {
    return dadd(dadd(dmul(ax, bx), dmul(ay, by)), dmul(az, bz));
}
__device__ __forceinline__ double d2r(const d3& p, double qx, double qy, double qz) {
    double dx = dsub(p.x, qx), dy = dsub(p.y, qy), dz = dsub(p.z, qz);
    return dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
}

// Whether a double is <= 0 or >= 0 by its bits: the FP64 pipe's comparisons cost as much as
// its additions. Not for NaN.
__device__ __forceinline__ bool le0(double v) { return __double_as_longlong(v) <= 0; }
__device__ __forceinline__ bool ge0(double v) {
    const long long b = __double_as_longlong(v);
    return b >= 0 || b == LLONG_MIN;
}

// The same values and regions as ericson() below in one path for a warp whose lanes lie in
// different regions: all six dot products, the region by the reference's tests in their
// order, then one division and one closest point with the region's operands selected (a
// term that a region does not have is skipped, not added as zero times something).
// ericson()'s seven exits, taken one after the other by a mixed warp, cost about twice the
// FP64 instructions, and this part issues one FP64 warp instruction per 16 cycles and SM.
__device__ __forceinline__ double ericson_sel(const d3& p, const d3& a, const d3& b, const d3& c,
                                              int* region) {
    const double abx = dsub(b.x, a.x), aby = dsub(b.y, a.y), abz = dsub(b.z, a.z);
    const double acx = dsub(c.x, a.x), acy = dsub(c.y, a.y), acz = dsub(c.z, a.z);
    const double apx = dsub(p.x, a.x), apy = dsub(p.y, a.y), apz = dsub(p.z, a.z);
    const double d1 = dot3r(abx, aby, abz, apx, apy, apz), d2 = dot3r(acx, acy, acz, apx, apy, apz);
    const double bpx = dsub(p.x, b.x), bpy = dsub(p.y, b.y), bpz = dsub(p.z, b.z);
    const double d3v = dot3r(abx, aby, abz, bpx, bpy, bpz), d4 = dot3r(acx, acy, acz, bpx, bpy, bpz);
    const double cpx = dsub(p.x, c.x), cpy = dsub(p.y, c.y), cpz = dsub(p.z, c.z);
    const double d5 = dot3r(abx, aby, abz, cpx, cpy, cpz), d6 = dot3r(acx, acy, acz, cpx, cpy, cpz);
    const double vc = dsub(dmul(d1, d4), dmul(d3v, d2));
    const double vb = dsub(dmul(d5, d2), dmul(d1, d6));
    const double va = dsub(dmul(d3v, d6), dmul(d5, d4));
    const double d43 = dsub(d4, d3v), d56 = dsub(d5, d6);  // their signs compare the two
    int g = 6;
    if (le0(va) && ge0(d43) && ge0(d56)) g = 5;
    if (le0(vb) && ge0(d2) && le0(d6)) g = 4;
    if (ge0(d6) && le0(d56)) g = 3;
    if (le0(vc) && ge0(d1) && le0(d3v)) g = 2;
    if (ge0(d3v) && le0(d43)) g = 1;
    if (le0(d1) && le0(d2)) g = 0;
    *region = g;
    // the nearest vertex's offset, or the region's first vertex
    double qx = g == 1 || g == 5 ? b.x : (g == 3 ? c.x : a.x);
    double qy = g == 1 || g == 5 ? b.y : (g == 3 ? c.y : a.y);
    double qz = g == 1 || g == 5 ? b.z : (g == 3 ? c.z : a.z);
    if (g == 2 || g >= 4) {
        // v = d1 / (d1 - d3), w = d2 / (d2 - d6), w = d43 / (d43 + d56), 1 / (va + vb + vc)
        const double num = g == 2 ? d1 : (g == 4 ? d2 : (g == 5 ? d43 : 1.0));
        const double x = g == 2 ? d1 : (g == 4 ? d2 : (g == 5 ? d43 : dadd(va, vb)));
        const double y = g == 2 ? -d3v : (g == 4 ? -d6 : (g == 5 ? d56 : vc));
        const double f = ddiv(num, dadd(x, y));
        const double s = g == 6 ? dmul(vb, f) : f;
        const double ux = g == 4 ? acx : (g == 5 ? dsub(c.x, b.x) : abx);
        const double uy = g == 4 ? acy : (g == 5 ? dsub(c.y, b.y) : aby);
        const double uz = g == 4 ? acz : (g == 5 ? dsub(c.z, b.z) : abz);
        qx = dadd(qx, dmul(s, ux));
        qy = dadd(qy, dmul(s, uy));
        qz = dadd(qz, dmul(s, uz));
        if (g == 6) {
            const double w = dmul(vc, f);
            qx = dadd(qx, dmul(acx, w));
            qy = dadd(qy, dmul(acy, w));
            qz = dadd(qz, dmul(acz, w));
        }
    }
    return d2r(p, qx, qy, qz);
}

static __device__ __noinline__ double ericson(const d3& p, const d3& a, const d3& b, const d3& c,
                                              int* region) {
    double abx = dsub(b.x, a.x), aby = dsub(b.y, a.y), abz = dsub(b.z, a.z);
    double acx = dsub(c.x, a.x), acy = dsub(c.y, a.y), acz = dsub(c.z, a.z);
    double apx = dsub(p.x, a.x), apy = dsub(p.y, a.y), apz = dsub(p.z, a.z);
    double d1 = dot3r(abx, aby, abz, apx, apy, apz), d2 = dot3r(acx, acy, acz, apx, apy, apz);
    if (d1 <= 0 && d2 <= 0) { *region = 0; return d2r(p, a.x, a.y, a.z); }
    double bpx = dsub(p.x, b.x), bpy = dsub(p.y, b.y), bpz = dsub(p.z, b.z);
    double d3v = dot3r(abx, aby, abz, bpx, bpy, bpz), d4 = dot3r(acx, acy, acz, bpx, bpy, bpz);
    if (d3v >= 0 && d4 <= d3v) { *region = 1; return d2r(p, b.x, b.y, b.z); }
    double vc = dsub(dmul(d1, d4), dmul(d3v, d2));
    if (vc <= 0 && d1 >= 0 && d3v <= 0) {
        double v = ddiv(d1, dsub(d1, d3v));
        *region = 2;
        return d2r(p, dadd(a.x, dmul(v, abx)), dadd(a.y, dmul(v, aby)), dadd(a.z, dmul(v, abz)));
    }
    double cpx = dsub(p.x, c.x), cpy = dsub(p.y, c.y), cpz = dsub(p.z, c.z);
    double d5 = dot3r(abx, aby, abz, cpx, cpy, cpz), d6 = dot3r(acx, acy, acz, cpx, cpy, cpz);
    if (d6 >= 0 && d5 <= d6) { *region = 3; return d2r(p, c.x, c.y, c.z); }
    double vb = dsub(dmul(d5, d2), dmul(d1, d6));
    if (vb <= 0 && d2 >= 0 && d6 <= 0) {
        double w = ddiv(d2, dsub(d2, d6));
        *region = 4;
        return d2r(p, dadd(a.x, dmul(w, acx)), dadd(a.y, dmul(w, acy)), dadd(a.z, dmul(w, acz)));
    }
    double va = dsub(dmul(d3v, d6), dmul(d5, d4));
    double d43 = dsub(d4, d3v), d56 = dsub(d5, d6);
    if (va <= 0 && d43 >= 0 && d56 >= 0) {
        double w = ddiv(d43, dadd(d43, d56));
        *region = 5;
        return d2r(p, dadd(b.x, dmul(w, dsub(c.x, b.x))), dadd(b.y, dmul(w, dsub(c.y, b.y))),
                   dadd(b.z, dmul(w, dsub(c.z, b.z))));
    }
    double denom = ddiv(1.0, dadd(dadd(va, vb), vc));
    double v = dmul(vb, denom), w = dmul(vc, denom);
    *region = 6;
    return d2r(p, dadd(dadd(a.x, dmul(abx, v)), dmul(acx, w)),
               dadd(dadd(a.y, dmul(aby, v)), dmul(acy, w)),
               dadd(dadd(a.z, dmul(abz, v)), dmul(acz, w)));
}

__device__ __forceinline__ void load_soup(const double* __restrict__ soup, int64_t t, d3& a, d3& b,
                                          d3& c) {
    const double2* r = reinterpret_cast<const double2*>(soup + t * kSoupStride);
    double2 v0 = __ldg(r), v1 = __ldg(r + 1), v2 = __ldg(r + 2), v3 = __ldg(r + 3), v4 = __ldg(r + 4);
    a = {v0.x, v0.y, v1.x};
    b = {v1.y, v2.x, v2.y};
    c = {v3.x, v3.y, v4.x};
}

// ------------------------------------------------------------------ FP32 record
// Translation-invariant FP32 data of a triangle (a, b, c), computed once from FP64, in
// the triangle's own orthonormal frame (u, v, n): u along b - a, v in the triangle's
// plane toward c, n = u x v. In that frame a = (0, 0), b = (bx, 0), c = (cx, cy) with
// cy >= 0, the triangle lies in the plane n = 0, and a point's squared distance is its
// squared in-plane distance to the 2-D triangle plus its squared n component. The frame
// is built by two Gram-Schmidt passes, so b and c lie in it to FP64 rounding even for
// slivers and collinear or repeated vertices (then v is any unit vector across u).
struct alignas(16) TriRec {
    float o0[3];       // a - centroid
    float nn[3];       // n
    float nerr;        // bound on |n (FP32) - n| (the plane test's normal error)
    float uu[3];       // u
    float vv[3];       // v
    float bx;          // |b - a|
    float cx, cy;      // c - a in the frame
    float e1x;         // (c - b) . u
    float ib;          // 1 / bx (0 if a == b)
    float inv1, inv2;  // 1 / |c - b|^2, 1 / |c - a|^2 (0 for a zero edge)
    float ok;          // 1: the face branch is allowed (bx > 0 and cy > 0)
    float pad_[3];
};
static_assert(sizeof(TriRec) == 96, "record layout");
constexpr float kRecNormalErr = 2.4e-7f;  // TriRec::nerr of every record
constexpr int kRecVec = static_cast<int>(sizeof(TriRec) / 16);  // float4 words per record

__device__ __forceinline__ void load_rec(const TriRec* __restrict__ recs, int t, TriRec& r) {
    const float4* s = reinterpret_cast<const float4*>(recs + t);
    float4* d = reinterpret_cast<float4*>(&r);
#pragma unroll
    for (int i = 0; i < kRecVec; ++i) d[i] = __ldg(s + i);
}

__device__ __forceinline__ float dot3f(float ax, float ay, float az, const float* b) {
    return fmaf(ax, b[0], fmaf(ay, b[1], __fmul_rn(az, b[2])));
}

// The point's offset from a, pa = (point - centroid) - (a - centroid), and its n
// component: the first steps of the distance, shared with the plane test.
struct PaN {
    float x, y, z, n;
};
__device__ __forceinline__ PaN pa_n(const TriRec& r, float dx, float dy, float dz) {
    PaN p;
    p.x = __fsub_rn(dx, r.o0[0]);
    p.y = __fsub_rn(dy, r.o0[1]);
    p.z = __fsub_rn(dz, r.o0[2]);
    p.n = dot3f(p.x, p.y, p.z, r.nn);
    return p;
}

// Squared FP32 distance from a point to the triangle, from pa_n; region numbered as the
// FP64 Ericson regions (0 a, 1 b, 2 ab, 3 c, 4 ac, 5 bc, 6 face). In the frame the
// point is (pu, pv, pn); it projects inside when the three 2-D edge functions
// (pv, (c - b) x (p - b), (a - c) x (p - c)) are >= 0 and the triangle has area, and
// is then at |pn|; otherwise its nearest point is on the boundary, at the smallest of
// the three 2-D segment distances (each with pn^2 added once at the end). Every lane
// measures all three segments: no branch splits a warp whose cells lie in different
// regions. Explicit intrinsics fix the operation sequence, so the value does not depend
// on whether the region is wanted (REG) or on the inlining context.
// Error (u = 2^-24, d the distance, e the largest centroid-to-vertex distance, r the
// sub-brick radius): pa errs by at most u (3 r + 4 d + 6 e) (the recentring, as
// before), |pa| <= d + 2 e; the frame rounded to FP32 and the three dots move the
// point by at most 7 u |pa|, the FP32 2-D vertices the triangle by 3 u e; the segment
// parameter, the residual and the sums add at most 7 u (d + 2 e), a face decision on
// the wrong side of an edge 4 u (d + 2 e): together below u (22 d + 39 e + 3 r), well
// inside the stated 48 u (d + 2 e + 2 r).
template <bool REG>
__device__ __forceinline__ float dist_rec_t(const TriRec& r, const PaN& p, int* reg) {
    const float pu = dot3f(p.x, p.y, p.z, r.uu), pv = dot3f(p.x, p.y, p.z, r.vv);
    const float qu1 = __fsub_rn(pu, r.bx);
    const float qu2 = __fsub_rn(pu, r.cx), qv2 = __fsub_rn(pv, r.cy);
    const float s1 = fmaf(r.e1x, pv, -__fmul_rn(r.cy, qu1));
    const float s2 = fmaf(r.cy, qu2, -__fmul_rn(r.cx, qv2));
    // a -> b along u
    const float t0 = __saturatef(__fmul_rn(pu, r.ib));
    const float r0u = fmaf(-t0, r.bx, pu);
    const float d0 = fmaf(r0u, r0u, __fmul_rn(pv, pv));
    // b -> c, direction (e1x, cy)
    const float t1 = __saturatef(__fmul_rn(fmaf(qu1, r.e1x, __fmul_rn(pv, r.cy)), r.inv1));
    const float r1u = fmaf(-t1, r.e1x, qu1), r1v = fmaf(-t1, r.cy, pv);
    const float d1 = fmaf(r1u, r1u, __fmul_rn(r1v, r1v));
    // c -> a, direction (-cx, -cy)
    const float t2 = __saturatef(__fmul_rn(-fmaf(qu2, r.cx, __fmul_rn(qv2, r.cy)), r.inv2));
    const float r2u = fmaf(t2, r.cx, qu2), r2v = fmaf(t2, r.cy, qv2);
    const float d2 = fmaf(r2u, r2u, __fmul_rn(r2v, r2v));
    const bool face = r.ok > 0.f && pv >= 0.f && s1 >= 0.f && s2 >= 0.f;
    float d = d0;
    int g = 0;
    if (REG) g = t0 <= 0.f ? 0 : (t0 >= 1.f ? 1 : 2);
    if (d1 < d) {
        d = d1;
        if (REG) g = t1 <= 0.f ? 1 : (t1 >= 1.f ? 3 : 5);
    }
    if (d2 < d) {
        d = d2;
        if (REG) g = t2 <= 0.f ? 3 : (t2 >= 1.f ? 0 : 4);
    }
    if (face) {
        d = 0.f;
        g = 6;
    }
    if (REG) *reg = g;
    return fmaf(p.n, p.n, d);
}

// The distance and its region.
__device__ __forceinline__ float dist_rec(const TriRec& r, float dx, float dy, float dz, int* reg) {
    return dist_rec_t<true>(r, pa_n(r, dx, dy, dz), reg);
}
// The distance alone (the same value as dist_rec).
__device__ __forceinline__ float dist_rec_val(const TriRec& r, float dx, float dy, float dz) {
    return dist_rec_t<false>(r, pa_n(r, dx, dy, dz), nullptr);
}

// The triangle's nearest point to a point (pa_n of it, the triangle's centroid at e from
// the same origin as the offsets): any point of the triangle to within 40u (d + 4e + 4r),
// d the distance; it need not be the nearest to the last bit.
__device__ __forceinline__ void nearest_point(const TriRec& r, const PaN& p, float ex, float ey,
                                              float ez, float& qx, float& qy, float& qz) {
    const float pu = dot3f(p.x, p.y, p.z, r.uu), pv = dot3f(p.x, p.y, p.z, r.vv);
    const float qu1 = pu - r.bx, qu2 = pu - r.cx, qv2 = pv - r.cy;
    const float t0 = __saturatef(pu * r.ib);
    const float t1 = __saturatef(fmaf(qu1, r.e1x, pv * r.cy) * r.inv1);
    const float t2 = __saturatef(-fmaf(qu2, r.cx, qv2 * r.cy) * r.inv2);
    float cu = t0 * r.bx, cv = 0.f;
    float d = fmaf(pu - cu, pu - cu, pv * pv);
    const float u1 = fmaf(t1, r.e1x, r.bx), v1 = t1 * r.cy;
    const float d1 = fmaf(pu - u1, pu - u1, (pv - v1) * (pv - v1));
    if (d1 < d) { d = d1; cu = u1; cv = v1; }
    const float u2 = fmaf(-t2, r.cx, r.cx), v2 = fmaf(-t2, r.cy, r.cy);
    const float d2 = fmaf(pu - u2, pu - u2, (pv - v2) * (pv - v2));
    if (d2 < d) { cu = u2; cv = v2; }
    if (r.ok > 0.f && pv >= 0.f && fmaf(r.e1x, pv, -r.cy * qu1) >= 0.f &&
        fmaf(r.cy, qu2, -r.cx * qv2) >= 0.f) {
        cu = pu;
        cv = pv;
    }
    qx = ex + r.o0[0] + fmaf(cu, r.uu[0], cv * r.vv[0]);
    qy = ey + r.o0[1] + fmaf(cu, r.uu[1], cv * r.vv[1]);
    qz = ez + r.o0[2] + fmaf(cu, r.uu[2], cv * r.vv[2]);
}

// sqrt to 2u (the pruning tests below carry wider margins).
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ------------------------------------------------------------------ box tests
// Which triangles can matter to some cell p of a box (half-widths hx, hy, hz and
// half-diagonal r around the origin), given one point q of the surface: p is at most
// b(p) = |p - q| + eps from the surface, so a triangle matters to p only when its lower
// bound is <= b(p) (eps carries the FP32 distances' errors). A triangle with centroid c and
// radius w lies in the ball of radius w around c and in its plane (unit normal n), that
// is in a disc, whose distance from p is (n . (p - c))^2 + max(0, lat - w)^2 squared, lat
// the in-plane distance of p from c. That is <= b^2 exactly when n . (p - c) <= b and
//     |p - c|^2 - b^2 <= w^2 + 2 w s,    s^2 = b^2 - (n . (p - c))^2,
// and the two quadratics leave |c|^2 - |q|^2 - 2 p . (c - q) on the left, linear in p: its
// minimum over the box is exact, where a test against the box's sphere gives away twice
// its radius along every direction. s^2 is bounded over the box by its value and gradient
// at the origin (its second-order part |p|^2 - (n . p)^2 is at most r^2). n = 0 (a
// degenerate triangle) leaves the ball test. Rounding: every term is formed from c, q, n and
// the box with relative errors that sum to less than 40u (|c|^2 + |q|^2 + r^2), the
// normal's own error nerr to less than 6 nerr (|c|^2 + r^2); `add` and the tests' own part of
// |c|^2 widen the right side by more. A comparison with a NaN keeps the triangle.
struct BoxTest {
    float qx, qy, qz, q2;
    float hx, hy, hz, r2;
    float e2;   // 2 eps (|q| + r) + eps^2, rounded up
    float qr;   // |q| + r + eps, rounded up (s <= qr without a plane)
    float add;  // absolute margin
};
__device__ __forceinline__ BoxTest box_test(float qx, float qy, float qz, float hx, float hy,
                                            float hz, float r, float eps, float pos) {
    BoxTest b;
    b.qx = qx; b.qy = qy; b.qz = qz;
    b.hx = hx; b.hy = hy; b.hz = hz;
    b.q2 = fmaf(qx, qx, fmaf(qy, qy, qz * qz));
    b.r2 = r * r;
    b.qr = (sqrtf(b.q2) + r + eps) * (1.f + 8.f * kU32);
    b.e2 = eps * (2.f * b.qr + eps) * (1.f + 8.f * kU32);
    // pos: absolute error of the positions beyond their own rounding
    b.add = fmaf(64.f * kU32, b.q2 + b.r2, 8.f * pos * (b.qr + pos)) + 1e-36f;
    return b;
}
// The test without the plane (s <= qr): false when no cell of the box can be concerned.
__device__ __forceinline__ bool box_ball(const BoxTest& b, float cx, float cy, float cz, float w,
                                         float pos) {
    const float c2 = fmaf(cx, cx, fmaf(cy, cy, cz * cz));
    const float g = fmaf(b.hx, fabsf(cx - b.qx), fmaf(b.hy, fabsf(cy - b.qy), b.hz * fabsf(cz - b.qz)));
    const float lin = fmaf(-2.f, g, c2 - b.q2);
    const float m = fmaf(64.f * kU32, c2, fmaf(8.f * pos, w, b.add));
    const float rhs = fmaf(w * (1.f + 32.f * kU32), fmaf(2.f, b.qr, w), b.e2) + m;
    return !(lin > rhs);
}
// The test with the plane; n.w bounds the error of the unit normal n.
__device__ __forceinline__ bool box_disc(const BoxTest& b, float cx, float cy, float cz, float w,
                                         const float4& n) {
    const float c2 = fmaf(cx, cx, fmaf(cy, cy, cz * cz));
    const float g = fmaf(b.hx, fabsf(cx - b.qx), fmaf(b.hy, fabsf(cy - b.qy), b.hz * fabsf(cz - b.qz)));
    const float lin = fmaf(-2.f, g, c2 - b.q2);
    const float m = fmaf(64.f * kU32 + 8.f * n.w, c2 + b.r2, fmaf(8.f * n.w, b.q2, b.add));
    const float nc = fmaf(n.x, cx, fmaf(n.y, cy, n.z * cz));
    const float gs = fmaf(b.hx, fabsf(fmaf(nc, n.x, -b.qx)),
                          fmaf(b.hy, fabsf(fmaf(nc, n.y, -b.qy)), b.hz * fabsf(fmaf(nc, n.z, -b.qz))));
    const float s2 = fmaf(2.f, gs, fmaf(-nc, nc, b.q2 + b.r2)) + (b.e2 + m);
    const float s = sqrt_approx(fmaxf(s2, 0.f));
    const float rhs = fmaf(w * (1.f + 32.f * kU32), fmaf(2.f, s, w), b.e2) + m;
    return !(s2 < 0.f) && !(lin > rhs);
}

// One cell's test against a disc: d the cell's offset from the centroid (squared length
// d2), pn its plane distance from the triangle, b its bound with the plane test's margin
// (plane_reach), w the triangle's radius or more (reach_term: w (1 + 20u) + 17u r). The
// offset's rounding moves d2 by at most 24u (b^2 + w^2) + 4u r (b + w), the right side's
// own by 8u (b^2 + w^2); b^2 exceeds the cell's bound squared by 136u b (b + 4e + 4r), w^2
// the radius squared by 40u w^2 + 34u w r.
__device__ __forceinline__ bool cell_disc(float d2, float pn, float b, float w) {
    const float s = sqrt_approx(fmaxf((b - fabsf(pn)) * (b + fabsf(pn)), 0.f));
    return fabsf(pn) <= b && !(d2 > fmaf(w, fmaf(2.f, s, w), b * b) * (1.f + 16.f * kU32));
}

// ------------------------------------------------------------------ outputs
struct Out {
    const uint8_t* occ;
    float* sdf32;
    double* sdf64;
    int* near_tri;
    uint8_t* near_reg;
    float* errbound;  // mixed: per-cell stated FP32 error bound (nullable)
};

__device__ __forceinline__ void write_cell(const Out& o, int64_t idx, double d, int tri, int reg) {
    const bool in = o.occ[idx] != 0;
    const double sd = in ? -d : d;
    if (o.sdf64) o.sdf64[idx] = sd;
    if (o.sdf32) o.sdf32[idx] = __double2float_rn(sd);
    if (o.near_tri) o.near_tri[idx] = tri;
    if (o.near_reg) o.near_reg[idx] = static_cast<uint8_t>(reg);
}

// Splits x (FP64) into hi = fl32(x) and lo = fl32(x - hi): hi + lo carries ~48
// bits, so differences of nearby points can be formed in FP32 without losing
// the bits that an FP32 subtraction of far-from-zero coordinates would drop.
__device__ __forceinline__ void split2(double x, float& hi, float& lo) {
    hi = __double2float_rn(x);
    lo = __double2float_rn(x - static_cast<double>(hi));
}

}  // namespace sdf
}  // namespace cmg::gpu
