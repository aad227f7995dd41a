// sdf_near.cu — distance per cell through an FP32 pass, one warp per 4^3 sub-brick.
//
// The brick candidate lists (k_brick_walk at brick edge 16) hold every triangle that
// can be nearest to some cell of the brick. A warp takes a sub-brick at a time from an
// LPT-ordered queue, two cells per lane (the same column, two layers apart), with no
// block-wide step:
//   1. probe: over the head of the brick list, the lanes' nearest triangles by
//      bounding sphere; their FP32 distances give the seed triangle, an upper bound U on
//      the sub-brick centre's distance and a surface point q near it;
//   2. filter: the brick list in steps of 192 (exact: 128); the entries that the ball test around q
//      keeps (box_ball) go to a short list in shared memory;
//   3. as soon as 32 of them wait, each lane loads one's record; those that the disc
//      test keeps (box_disc) are staged in shared memory, and every cell tests them
//      (cell_disc); the (cell, triangle) pairs left are evaluated 32 at a time, one per
//      lane (a triangle that some cell needs is needed by 8 to 18 of the 64);
//   4. near-ties (FP32 distance within twice the stated error of the cell's minimum) are
//      kept as (cell, triangle) pairs, and the FP64 distance in the reference's order is
//      taken over the pairs, one per lane: for every cell (kPrecExact, the reference's
//      bits), or for the cells within `band` cells of the surface (kPrecMixed).
// Centroids are stored as FP32 hi + lo pairs relative to the grid corner, so the
// centroid-to-centre differences are formed in FP32 without losing the low bits (the
// sub-brick recentring).
#include <cuda_runtime.h>
#include <math_constants.h>

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

constexpr int kWarps = 4;       // independent warps per CTA
// List entries per lane and scan step (loads in flight): the exact kernel's FP64 part leaves
// fewer registers (231x247x256, mixed / exact, ms: 4 entries 4.41 / 6.95, 5: 4.39 / 6.97, 6:
// 4.36 / 7.10, 8: 4.45 / 7.38).
template <int PREC>
constexpr int kSteps = PREC == kPrecMixed ? 6 : 4;
constexpr int kWait = 32 * (kSteps<kPrecMixed> + 1);  // entries that can wait for the disc test
constexpr int kPairs = 256;     // near-tie pairs kept per sub-brick
constexpr int kSkip = 512;      // of longer lists the probe reads every other step
constexpr float kItemCost = 1024.f;  // a sub-brick's fixed work, in list entries
constexpr float kHeavy = 0.25f;      // lists over this part of a warp's share are shared
constexpr unsigned kAll = 0xffffffffu;
constexpr float kKept = -2.f;  // the distance of a near-tie pair that no threshold drops

struct WarpMem {
    // staged records, their centroids (radius widened: reach_term) and ids
    TriRec rec[32];
    float4 c[32];
    int t[32];
    // per cell: its FP32 minimum (bits of the squared distance, then the triangle), and the
    // plane_reach of its bound (-1: not a cell of the grid)
    unsigned long long best[64];
    float reach[64];
    float pos[12];  // cell offsets from the sub-brick centre, per axis
    unsigned short ev[96];  // (cell, staged triangle) pairs that wait: cell | triangle << 6
    // FP64 results per cell: the smallest squared distance (bits) and, for it, the smallest
    // (triangle << 3) | region
    unsigned long long d[64], win[64];
    double ctr[12];  // FP64 cell centres of the sub-brick, per axis
    float thr2[64];  // per cell: keeps near-ties up to this squared FP32 distance
    // of the sub-brick, the same for all lanes (kept out of registers):
    BoxTest box;
    float4 mid[2];  // its centre from the grid corner, FP32 hi and lo; mid[0].w: its radius r
    float4 off;     // its centre from the brick's; w: the list's position error
    float4 con;     // x: kap, y: kapx, z: ebr4, w: keep2 (sub_brick)
    int org[3];     // its first cell
    unsigned long long evals, filtered, evals64, bandc;  // this warp's counters
    int wait[kWait];  // list entries that passed the ball test
    // near-tie pairs: triangle, FP32 squared distance, cell
    int pt[kPairs];
    float pd[kPairs];
    unsigned char pc[kPairs];
};

// Drops the pairs beyond their cells' thresholds (which only fall); the number kept.
__device__ __noinline__ int prune(WarpMem& M, int n) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    __syncwarp();
    int kept = 0;
#pragma unroll 1
    for (int k0 = 0; k0 < n; k0 += 32) {
        const bool in = k0 + lane < n;
        const int k = in ? k0 + lane : 0;
        const int t = M.pt[k], c = M.pc[k];
        const float d = M.pd[k];
        const bool live = in && d <= M.thr2[c];
        const unsigned m = __ballot_sync(kAll, live);
        __syncwarp();
        if (live) {
            const int to = kept + __popc(m & below);
            M.pt[to] = t;
            M.pd[to] = d;
            M.pc[to] = static_cast<unsigned char>(c);
        }
        kept += __popc(m);
        __syncwarp();
    }
    return kept;
}

// What a CTA's warps exchange about a shared sub-brick.
struct Shared {
    unsigned long long grab;
    unsigned u[kWarps];
    int seed[kWarps];
    int npair[kWarps];
};

// The FP64 distance of one pair per lane (in: there is one) into the cells' results.
__device__ __forceinline__ void refine_32(WarpMem& M, const double* __restrict__ soup, int t, int c, bool in) {
    d3 a, b, cc;
    load_soup(soup, t, a, b, cc);
    int reg;
    const double e2 = ericson_sel(d3{M.ctr[c & 3], M.ctr[4 + ((c >> 2) & 3)], M.ctr[8 + (c >> 4)]}, a, b, cc, &reg);
    // (a NaN or infinite distance counts for nothing)
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(e2));
    const bool use = in && e2 <= DBL_MAX;
    const unsigned long long was = M.d[c];
    __syncwarp();
    if (use && bits < was) atomicMin(&M.d[c], bits);
    __syncwarp();
    const unsigned long long now = M.d[c];
    if (now != was) M.win[c] = ~0ull;
    __syncwarp();
    if (use && bits == now) atomicMin(&M.win[c], (static_cast<unsigned long long>(t) << 3) | static_cast<unsigned>(reg));
    __syncwarp();
}

// The FP64 distances of the n pairs, one per lane: the smallest, by the lowest triangle on
// ties. A pair that later turns out to lie beyond its cell's final threshold changes
// nothing: the minimum over more triangles is the same.
__device__ __noinline__ void refine(WarpMem& M, int n, const double* __restrict__ soup) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k0 = 0; k0 < n; k0 += 32) {
        const bool in = k0 + lane < n;
        const int k = in ? k0 + lane : n - 1;
        refine_32(M, soup, M.pt[k], M.pc[k], in);
    }
}

// The same for the pairs of all the CTA's warps (S.npair each): of every 128 in a row, this
// warp's 32.
__device__ __noinline__ void refine_shared(WarpMem& M, const WarpMem* all, const Shared& S,
                                           const double* __restrict__ soup) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int w = 0; w < kWarps; ++w) n += S.npair[w];
#pragma unroll 1
    for (int k0 = threadIdx.x & ~31; k0 < n; k0 += 32 * kWarps) {
        const bool in = k0 + lane < n;
        int k = in ? k0 + lane : n - 1, w = 0;
        while (k >= S.npair[w]) k -= S.npair[w++];
        refine_32(M, soup, all[w].pt[k], all[w].pc[k], in);
    }
}

// A triangle's centroid relative to the sub-brick centre, from its hi + lo pair.
__device__ __forceinline__ float4 recentre(const float4& hi, const float4& lo, const float4& mh, const float4& ml) {
    return make_float4((hi.x - mh.x) + (lo.x - ml.x), (hi.y - mh.y) + (lo.y - ml.y), (hi.z - mh.z) + (lo.z - ml.z),
                       hi.w);
}

// Reach of a cell's test against a triangle: w (1 + 20u) + 17u r, rounded up (w the
// triangle's radius, r the sub-brick radius; the margins cover the FP32 rounding of the
// centroids and cell offsets).
__device__ __forceinline__ float reach_term(float w, float r) {
    return __fmaf_ru(w, 1.f + 20.f * kU32, __fmul_ru(17.f * kU32, r));
}

// A cell's bound, from its smallest FP32 squared distance so far, d2: a near-tie's FP32
// distance is within two stated errors of the cell's FP32 minimum m = sqrt(d2) and its
// true distance d one more, so d <= m + 3 E(d), E(d) = 48u (d + 2e + 2r), which gives
// 3 E(d) <= 144.1u m + 288.2u (e + r); with the square root's rounding,
// sqrt(d2)(1 + 160u) + kapx, kapx = RU(300u (e + r) + 4 kTinyDist), covers it (each of the
// errors has kTinyDist besides, the ends of FP32's range). So the FP32 pass
// evaluates every triangle that can be the FP32 minimum or a near-tie of it, whatever
// order the candidates come in: the cell ends with the exact (FP32 distance, triangle
// id) minimum over all triangles, independent of which candidates the walk listed.
__device__ __forceinline__ float cell_bound_x(float d2, float kapx) {
    return __fmaf_ru(sqrt_approx(d2), 1.f + 160.f * kU32, kapx);
}

// The near-tie threshold of a cell whose FP32 minimum is sqrt(d2), squared and rounded
// up: at least (m + 2 eb)^2, eb = 48u (m + 2e + 2r) + kTinyDist the stated bound (kap =
// 98u (e + r) + kTinyDist).
__device__ __forceinline__ float near_thr2(float d2, float kap) {
    const float thr = __fmaf_ru(sqrt_approx(d2), 1.f + 100.f * kU32, __fmul_ru(2.f, kap));
    return __fmul_ru(thr, thr);
}

// Largest computed plane distance |n . (cell - a)| of a triangle that can still reach
// the cell's bound b: such a triangle is within b of the cell, so |cell - a| <= b + 2e (a
// a vertex, e the mesh's largest centroid-to-vertex distance), and the FP32 plane
// distance errs by at most nerr |cell - a| (nerr bounds the FP32 unit normal's error, the
// same for every record) plus the rounding of the recentred offsets and the dot
// product, all within (nerr + 64u)(b + 4e + 4r) (ebr4 = 4(e + r), rounded up).
__device__ __forceinline__ float plane_reach(float b, float ebr4) {
    return __fmaf_ru(__fadd_ru(b, ebr4), __fadd_ru(kRecNormalErr, 64.f * kU32), b);
}

// A cell's FP32 minimum as one number: the smaller distance, the lower triangle on ties.
__device__ __forceinline__ unsigned long long near_key(float d2, int t) {
    return (static_cast<unsigned long long>(__float_as_uint(d2)) << 32) | static_cast<unsigned>(t);
}
__device__ __forceinline__ float key_dist(unsigned long long k) { return __uint_as_float(static_cast<unsigned>(k >> 32)); }
__device__ __forceinline__ int key_tri(unsigned long long k) { return static_cast<int>(static_cast<unsigned>(k)); }

// Lowers a nonnegative float (several lanes may).
__device__ __forceinline__ void lower(float* at, float v) {
    atomicMin(reinterpret_cast<unsigned*>(at), __float_as_uint(v));
}

// What the kernel reads and writes.
struct Args {
    const MeshSeg* segs;
    int nseg;
    const uint32_t* work;
    int64_t nwork;
    int grab_n, probe_n;
    const double* soup;
    const float4 *tinfo, *tinfo_lo;
    const TriRec* trec;
    const int64_t* cand_rng;
    const int* cand;
    const float4* cand_c;
    float band_cells;
    Out o;
};

// One sub-brick: by this warp alone, or (COOP) by the CTA's warps together, each over its
// part of the list. item: sub-brick of the queue.
//
// THIN: the meshes have triangles without a face in their records (repeated or collinear
// corners, or thinner than a billionth). For those the reference's FP64 operations may give no
// number (0 / 0; the triangle then counts for nothing) or one that is not the distance. So they
// are no seeds, lower no cell's minimum and bound (nor the walk's), and every one that might be
// nearest to a cell goes to FP64, which decides. Meshes without any, by far the most, keep the
// kernel without it (2 % faster in mixed precision).
template <int PREC, bool THIN, bool COOP>
__device__ __forceinline__ void sub_brick(const Args& g, const int64_t item, WarpMem& M, Shared& S,
                                          const WarpMem* all) {
    constexpr bool EXACT = PREC == kPrecExact;
    constexpr int kStep = kSteps<PREC>;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int64_t gb = g.work[item >> 6];  // the bricks in order, 64 sub-bricks each
    const MeshSeg& s = g.segs[find_seg<&MeshSeg::brick_begin>(g.segs, g.nseg, gb)];
    float px, py, zA, zB;  // the lane's two cells, lane and 32 + lane
    bool okA, okB;         // are cells of the grid and the slab
    // ---- geometry: each lane forms one number per axis in FP64 (the FP64 pipe takes 16 cycles
    //      per warp instruction), the others get it by shuffles
    float hx, hy, hz;
    {
        const SubGeo q = sub_geo(s, gb - s.brick_begin, static_cast<int>(item & 63));
        if (q.empty) return;
        const double h = s.g.h;
        const int a = lane < 12 ? lane >> 2 : min(lane - 12, 2), i = lane & 3;
        const int lo = a == 0 ? q.x0 : (a == 1 ? q.y0 : q.z0);
        const int hi = a == 0 ? q.x1 : (a == 1 ? q.y1 : q.z1);
        const double ck = 0.5 * (lo + hi) * h;  // the sub-brick centre from the corner
        const float pv = static_cast<float>(fma(lo + i + 0.5, h, -ck));
        const float hw = __double2float_ru(0.5 * (hi - lo - 1) * h);
        float ch, cl;
        split2(ck, ch, cl);
        px = __shfl_sync(kAll, pv, lane & 3);
        py = __shfl_sync(kAll, pv, 4 + ((lane >> 2) & 3));
        zA = __shfl_sync(kAll, pv, 8 + (lane >> 4));
        zB = __shfl_sync(kAll, pv, 10 + (lane >> 4));
        hx = __shfl_sync(kAll, hw, 12);
        hy = __shfl_sync(kAll, hw, 13);
        hz = __shfl_sync(kAll, hw, 14);
        if (lane < 12) {
            M.ctr[lane] = cell_center(s.g.corner[a], lo + i, h);
            M.pos[lane] = pv;
        } else if (lane < 15) {
            // the list's centroids are relative to the brick's centre, without their lo parts
            const int b0 = lo / s.brick * s.brick;
            const int n = a == 0 ? s.g.nx : (a == 1 ? s.g.ny : s.g.nz);
            const float bc = span_centre(b0, min(b0 + s.brick, n), static_cast<float>(h));
            (&M.mid[0].x)[a] = ch;
            (&M.mid[1].x)[a] = cl;
            (&M.off.x)[a] = (ch - bc) + cl;
            M.org[a] = lo;
        }
        const int x = q.x0 + (lane & 3), y = q.y0 + ((lane >> 2) & 3), z = q.z0 + (lane >> 4);
        const bool col = x < q.x1 && y < q.y1;
        okA = col && z < q.z1 && z >= s.g.z0 && z < s.g.z1;
        okB = col && z + 2 < q.z1 && z + 2 >= s.g.z0 && z + 2 < s.g.z1;
    }
    const float emax = s.emax_all;
    {
        const float r = __fsqrt_ru(__fmaf_ru(hx, hx, __fmaf_ru(hy, hy, __fmul_ru(hz, hz))));
        // the stated FP32 error of a distance near d is 48u (d + 2e + 2r); kap carries its
        // constant part, kapx that of the cells' bounds (three of them)
        const float er = __fadd_ru(emax, r);
        const float kap = __fmaf_ru(98.f * kU32, er, kTinyDist);
        // mixed: near-ties beyond what a band cell can reach are not kept
        float keep2 = FLT_MAX;
        if (!EXACT) {
            const float bh = g.band_cells * static_cast<float>(s.g.h);
            const float far =
                fmaxf(0.f, __fmaf_ru(fabsf(bh), 512.f * kU32, bh + 16.f * kap) * (1.f + 8.f * kU32));
            keep2 = far * far * (1.f + 8.f * kU32);
        }
        M.thr2[lane] = okA ? keep2 : -1.f;
        M.thr2[32 + lane] = okB ? keep2 : -1.f;
        M.reach[lane] = okA ? FLT_MAX : -1.f;
        M.reach[32 + lane] = okB ? FLT_MAX : -1.f;
        M.best[lane] = M.best[32 + lane] = near_key(FLT_MAX, INT_MAX);
        M.d[lane] = M.d[32 + lane] = static_cast<unsigned long long>(__double_as_longlong(DBL_MAX));
        M.win[lane] = M.win[32 + lane] = static_cast<unsigned long long>(INT_MAX) << 3;
        __syncwarp();  // the last sub-brick's reads of these are done
        if (lane == 0) {
            M.mid[0].w = r;
            M.off.w = list_tol(s.scale);
            M.con = make_float4(kap, __fmaf_ru(300.f * kU32, er, 4.f * kTinyDist), __fmul_ru(4.f, er), keep2);
        }
        __syncwarp();
    }
    const int64_t c0 = g.cand_rng[2 * gb];
    const int nc = static_cast<int>(g.cand_rng[2 * gb + 1] - c0);
    const int* __restrict__ list = g.cand + c0;
    const float4* __restrict__ listc = g.cand_c + c0;
    // (the warps of a shared sub-brick take every fourth 32 entries)
    constexpr int kNext = COOP ? 32 * kWarps : 32;
    const int first = COOP ? wid * 32 : 0;
    constexpr int step = kNext * kStep;

    // ---- 1. probe: per lane, over the list's head, the triangle of the nearest centroid
    //         and the one of the smallest power distance |c|^2 - w^2 (w the radius: large
    //         triangles near the centre); then their FP32 distances
    float U = FLT_MAX;
    int seed = INT_MAX;
    {
        const float4 off = M.off;
        float bestc = FLT_MAX, bestp = FLT_MAX;
        int kc = -1, kp = -1;
        const int np = min(nc, g.probe_n);
        const int skip = np > kSkip ? 2 * step : step;
        for (int k0 = first + lane; k0 < np; k0 += skip) {
            float4 e[kStep];
#pragma unroll
            for (int i = 0; i < kStep; ++i)
                e[i] = k0 + kNext * i < np ? __ldg(listc + k0 + kNext * i) : make_float4(FLT_MAX, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kStep; ++i) {
                const float ex = e[i].x - off.x, ey = e[i].y - off.y, ez = e[i].z - off.z;
                const float c2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez)), pw = fmaf(-e[i].w, e[i].w, c2);
                if (c2 < bestc) { bestc = c2; kc = k0 + kNext * i; }
                if (pw < bestp) { bestp = pw; kp = k0 + kNext * i; }
            }
        }
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            const int at = k == 0 ? kc : kp;
            if (at >= 0 && (k == 0 || kp != kc)) {
                const int t = list[at];
                TriRec r;
                load_rec(g.trec, t, r);
                if (THIN && !(r.ok > 0.f)) continue;
                const float4 e = recentre(g.tinfo[t], g.tinfo_lo[t], M.mid[0], M.mid[1]);
                const float dc = sqrt_approx(fmaf(e.x, e.x, fmaf(e.y, e.y, e.z * e.z)));
                const float d = sqrt_approx(dist_rec_val(r, -e.x, -e.y, -e.z));
                const float ub = d * (1.f + 32.f * kU32) + (32.f * kU32 * (dc + 2.f * e.w) + kTinyDist);
                if (ub < U || (ub == U && t < seed)) { U = ub; seed = t; }
            }
        }
        const unsigned m = __reduce_min_sync(kAll, __float_as_uint(U));
        seed = __reduce_min_sync(kAll, __float_as_uint(U) == m ? seed : INT_MAX);
        U = __uint_as_float(m);
        if (COOP) {
            if (lane == 0) {
                S.u[wid] = __float_as_uint(U);
                S.seed[wid] = seed;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kWarps; ++k) {
                const float u = __uint_as_float(S.u[k]);
                const int t = S.seed[k];
                if (u < U || (u == U && t < seed)) { U = u; seed = t; }
            }
        }
    }

    // ---- the seed: every cell's first bound, and the box test around its nearest point to
    //      the centre (eps: four stated errors of the FP32 distances, and q's own)
    int npair = 0, nfull = 0, neval = 0, nstaged = 0;  // nfull: pairs refined before the end
    // appends near-ties of triangle t, one of each lane in m; there is room
    auto push = [&](unsigned m, int t, float d, int cell) {
        if ((m >> lane) & 1u) {
            const int k = npair + __popc(m & below);
            M.pt[k] = t;
            M.pd[k] = d;
            M.pc[k] = static_cast<unsigned char>(cell);
        }
        npair += __popc(m);
    };
    // a cell's minimum, and what follows from it, after a triangle's distance
    auto improve = [&](int cell, float d, int t) {
        const unsigned long long key = near_key(d, t), was = M.best[cell];
        if (key >= was) return;
        atomicMin(&M.best[cell], key);
        if (d < key_dist(was)) {
            const float4 con = M.con;
            lower(&M.reach[cell], plane_reach(cell_bound_x(d, con.y), con.z));
            lower(&M.thr2[cell], near_thr2(d, con.x));
        }
    };
    if (seed != INT_MAX) {
        const float4 con = M.con;
        const float4 e = recentre(g.tinfo[seed], g.tinfo_lo[seed], M.mid[0], M.mid[1]);
        TriRec r;
        load_rec(g.trec, seed, r);
        float qx, qy, qz;
        nearest_point(r, pa_n(r, -e.x, -e.y, -e.z), e.x, e.y, e.z, qx, qy, qz);
        const BoxTest b =
            box_test(qx, qy, qz, hx, hy, hz, M.mid[0].w,
                     __fmaf_ru(240.f * kU32, U + 4.f * M.mid[0].w, fmaf(40.f * kU32, con.z, 4.f * con.x)), M.off.w);
        if (lane == 0) M.box = b;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            const int cell = lane + 32 * half;
            const bool ok = half ? okB : okA;
            const float d = dist_rec_val(r, px - e.x, py - e.y, (half ? zB : zA) - e.z);
            if (ok) improve(cell, d, seed);
            const unsigned m = __ballot_sync(kAll, ok && d <= M.thr2[cell]);
            if (!COOP || wid == 0) push(m, seed, d, cell);
        }
        neval = 64;
    }
    __syncwarp();

    // ---- 2 + 3. filter, disc test, evaluation
    int nwait = 0, cur = first;
    while (cur < nc || nwait > 0) {
        if (cur < nc && nwait < 32) {
            const BoxTest box = M.box;
            const float4 off = M.off;
            float4 e[kStep];
#pragma unroll
            for (int i = 0; i < kStep; ++i)
                e[i] = cur + lane + kNext * i < nc ? __ldg(listc + cur + lane + kNext * i)
                                                : make_float4(CUDART_NAN_F, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kStep; ++i) {
                const float ex = e[i].x - off.x, ey = e[i].y - off.y, ez = e[i].z - off.z;
                // without a seed nothing is known: every triangle with a place
                const bool take = seed != INT_MAX ? ex == ex && box_ball(box, ex, ey, ez, e[i].w, off.w)
                                                  : ex * ex + ey * ey + ez * ez <= FLT_MAX;
                const unsigned m = __ballot_sync(kAll, take);
                if (take) M.wait[nwait + __popc(m & below)] = cur + lane + kNext * i;
                nwait += __popc(m);
            }
            cur += step;
            if (nwait < 32 && cur < nc) continue;
        }
        __syncwarp();
        // the last 32 waiting (all of them at the end of the list): one per lane
        const int take_n = min(nwait, 32);
        nwait -= take_n;
        int staged;
        {
            bool live = lane < take_n;
            const int t = live ? list[M.wait[nwait + lane]] : -1;
            TriRec r;
            float4 e;
            if (live) {
                e = recentre(g.tinfo[t], g.tinfo_lo[t], M.mid[0], M.mid[1]);
                load_rec(g.trec, t, r);
                if (seed != INT_MAX)
                    live = t != seed && box_disc(M.box, e.x, e.y, e.z, e.w,
                                                 make_float4(r.nn[0], r.nn[1], r.nn[2], kRecNormalErr));
            }
            const unsigned m = __ballot_sync(kAll, live);
            staged = __popc(m);
            if (live) {
                const int pos = __popc(m & below);
                M.rec[pos] = r;
                M.c[pos] = make_float4(e.x, e.y, e.z, reach_term(e.w, M.mid[0].w));
                M.t[pos] = THIN && !(r.ok > 0.f) ? ~t : t;
            }
        }
        __syncwarp();
        nstaged += staged;
        int nev = 0;
        for (int j = 0; j <= staged; ++j) {
            if (j < staged) {
                const float4 c = M.c[j];
                const TriRec& R = M.rec[j];
                const float dx = px - c.x, dy = py - c.y, dzA = zA - c.z, dzB = zB - c.z;
                const float xy = fmaf(dx, dx, dy * dy);
                // a triangle no nearer than its disc, which lies beyond the cell's bound, is
                // skipped; the others are evaluated cell by cell
                const bool a = cell_disc(fmaf(dzA, dzA, xy), pa_n(R, dx, dy, dzA).n, M.reach[lane], c.w);
                const bool b = cell_disc(fmaf(dzB, dzB, xy), pa_n(R, dx, dy, dzB).n, M.reach[32 + lane], c.w);
                const unsigned mA = __ballot_sync(kAll, a), mB = __ballot_sync(kAll, b);
                if (!(mA | mB)) continue;
                if (a) M.ev[nev + __popc(mA & below)] = static_cast<unsigned short>(lane | j << 6);
                nev += __popc(mA);
                if (b) M.ev[nev + __popc(mB & below)] = static_cast<unsigned short>(32 | lane | j << 6);
                nev += __popc(mB);
            }
            while (nev >= 32 || (j == staged && nev > 0)) {
                __syncwarp();
                const int n = min(nev, 32);
                nev -= n;
                const bool in = lane < n;
                const int pr = M.ev[nev + (in ? lane : 0)], cell = pr & 63, k = pr >> 6;
                const float4 c = M.c[k];
                const int t = M.t[k];
                const float d = dist_rec_val(M.rec[k], M.pos[cell & 3] - c.x, M.pos[4 + ((cell >> 2) & 3)] - c.y,
                                             M.pos[8 + (cell >> 4)] - c.z);
                neval += n;
                const bool face = !THIN || t >= 0;
                if (in && face) improve(cell, d, t);
                __syncwarp();
                float thr = M.thr2[cell];
                if (!EXACT && !face) thr = near_thr2(key_dist(M.best[cell]), M.con.x);  // beyond the band too
                const unsigned m = __ballot_sync(kAll, in && d <= thr);
                if (m) {
                    if (npair + 32 > kPairs) {
                        npair = prune(M, npair);
                        if (npair + 32 > kPairs) {
                            refine(M, npair, g.soup);
                            nfull += npair;
                            npair = 0;
                        }
                    }
                    push(m, face ? t : ~t, EXACT || face ? d : kKept, cell);
                }
            }
        }
        __syncwarp();
    }
    unsigned long long bestA = M.best[lane], bestB = M.best[32 + lane];
    if (COOP) {  // the minima over the warps' parts of the list
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kWarps; ++k) {
            bestA = min(bestA, all[k].best[lane]);
            bestB = min(bestB, all[k].best[32 + lane]);
        }
        const float4 con = M.con;
        if (okA) M.thr2[lane] = fminf(near_thr2(key_dist(bestA), con.x), con.w);
        if (okB) M.thr2[32 + lane] = fminf(near_thr2(key_dist(bestB), con.x), con.w);
        __syncwarp();
    }

    // ---- 4. FP64 distances of the near-ties: every cell's (exact), or the band cells'
    const float d32A = sqrtf(key_dist(bestA)), d32B = sqrtf(key_dist(bestB));
    // the mesh's largest triangle radius (not the brick's candidates', which depend on the
    // candidate walk): the bound, and the band it selects, are the same whatever slab of
    // the grid is evaluated
    const float er2 = 2.f * emax + 2.f * M.mid[0].w;
    const float bh = g.band_cells * static_cast<float>(s.g.h);
    const float ebA = 48.f * kU32 * (d32A + er2) + kTinyDist, ebB = 48.f * kU32 * (d32B + er2) + kTinyDist;
    const bool fineA = okA && (EXACT || d32A <= bh + ebA);
    const bool fineB = okB && (EXACT || d32B <= bh + ebB);
    const unsigned maskA = __ballot_sync(kAll, fineA), maskB = __ballot_sync(kAll, fineB);
    if ((maskA | maskB) || (THIN && !EXACT)) {
        if (!EXACT) {  // the near-ties of the band's cells only
            if (!fineA) M.thr2[lane] = -1.f;
            if (!fineB) M.thr2[32 + lane] = -1.f;
        }
        npair = prune(M, npair);
        if (COOP) {
            if (lane == 0) S.npair[wid] = npair;
            __syncthreads();
            refine_shared(M, all, S, g.soup);
        } else if (npair > 0) {
            refine(M, npair, g.soup);
        }
    }
    const bool full = COOP ? __syncthreads_or(nfull) != 0 : nfull != 0;
    if (lane == 0) {
        M.evals += neval;
        M.filtered += nstaged;
        M.evals64 += npair + nfull;
        if ((!EXACT || full) && !(COOP && wid)) M.bandc += __popc(maskA) + __popc(maskB);
    }
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
        if (!(half ? okB : okA) || (COOP && half != wid)) continue;
        const int x = M.org[0] + (lane & 3), y = M.org[1] + ((lane >> 2) & 3), z = M.org[2] + (lane >> 4) + 2 * half;
        const int64_t idx = s.vox_begin + (static_cast<int64_t>(z - s.g.z0) * s.g.ny + y) * s.g.nx + x;
        if (half ? fineB : fineA) {
            unsigned long long d = M.d[lane + 32 * half], win = M.win[lane + 32 * half];
            if (COOP) {
#pragma unroll
                for (int k = 0; k < kWarps; ++k) {
                    const unsigned long long d2 = all[k].d[lane + 32 * half], w2 = all[k].win[lane + 32 * half];
                    if (d2 < d || (d2 == d && w2 < win)) { d = d2; win = w2; }
                }
            }
            write_cell(g.o, idx, __dsqrt_rn(__longlong_as_double(static_cast<long long>(d))),
                       static_cast<int>(win >> 3), static_cast<int>(win & 7u));
            if (g.o.errbound) g.o.errbound[idx] = 0.f;
        } else {
            const int t = key_tri(half ? bestB : bestA);
            int reg = 0;
            if (THIN && !EXACT) {  // a nearer triangle without a face
                unsigned long long d = M.d[lane + 32 * half], win = M.win[lane + 32 * half];
                if (COOP) {
#pragma unroll
                    for (int k = 0; k < kWarps; ++k) {
                        const unsigned long long d2 = all[k].d[lane + 32 * half], w2 = all[k].win[lane + 32 * half];
                        if (d2 < d || (d2 == d && w2 < win)) { d = d2; win = w2; }
                    }
                }
                const double e = __dsqrt_rn(__longlong_as_double(static_cast<long long>(d)));
                if (e < static_cast<double>(half ? d32B : d32A) && !(g.trec[win >> 3].ok > 0.f)) {
                    write_cell(g.o, idx, e, static_cast<int>(win >> 3), static_cast<int>(win & 7u));
                    if (g.o.errbound) g.o.errbound[idx] = half ? ebB : ebA;
                    continue;
                }
            }
            if (g.o.near_reg && t != INT_MAX) {
                // the region of the nearest triangle: its distance again, recentred exactly
                // as before (the same value, now with the region)
                const float4 e = recentre(g.tinfo[t], g.tinfo_lo[t], M.mid[0], M.mid[1]);
                TriRec r;
                load_rec(g.trec, t, r);
                dist_rec(r, px - e.x, py - e.y, (half ? zB : zA) - e.z, &reg);
            }
            write_cell(g.o, idx, static_cast<double>(half ? d32B : d32A), t, reg);
            if (g.o.errbound) g.o.errbound[idx] = half ? ebB : ebA;
        }
    }
    if (COOP) __syncthreads();  // the others' results are read before they are set again
    else __syncwarp();
}

// Registers are budgeted for 5 CTAs (20 warps) per SM: 96 a thread (231x247x256 surface,
// exact / mixed: 7.0 / 4.4 ms; 4 CTAs at 128: 7.2 / 4.6, 6 at 80: 8.2 / 6.1, spills).
// Pairs one per lane instead of triangles for all 64 cells, and the probe's skipping (a seed
// from half of a long list loosens the bound a little: 4 % more triangles are staged), for
// 137^3 around 128k triangles, exact: 2.48 -> 2.21 -> 2.12 ms; 118x126x130 around 65k, mixed:
// 1.40 -> 1.26 -> 1.24; 24 meshes, mixed: 11.2 -> 10.7 -> 10.5; the first grid: 1 to 2 %.
// A quarter of the list lost 10 %.
// grab_n: consecutive sub-bricks taken from the queue at once (they share one brick list).
// probe_n: entries of the brick list the probe scans: all of it unless asked for less (the
// 128^3 grid around 65k triangles: 1.4 ms; a head of 2048 leaves the sub-bricks with the
// longest lists a loose bound, 7.1 ms before they were shared).
// The queue's first sub-bricks, those whose lists are long beside a warp's share of all the
// work, are shared by a CTA's warps, each taking a quarter of the list (the minima over the
// parts are the minimum over the list); the lists get shorter (to within an eighth), so the
// first light one ends the sharing. With few sub-bricks in all, every one is shared. (128^3 grid around 65k
// triangles: 3.1 -> 1.4 ms, the warp with the longest list had ended last; 63^3 around 1280
// triangles, all shared: 0.28 -> 0.19 ms.) Their lists are dealt out by 32 entries, and the
// pairs for FP64 by 32 pairs, whichever warp found them: with parts of 128 entries and
// everybody's own pairs, half of a shared sub-brick's time was waiting for the last warp (63^3:
// 0.19 -> 0.17 ms, 35^3 around 320 triangles: 0.11 -> 0.075 ms).
template <int PREC, bool THIN>
__global__ void __launch_bounds__(32 * kWarps, 5)
k_sdf_near(const Args g, unsigned long long* __restrict__ queue, Stats* __restrict__ st) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ Shared S;
    WarpMem* const all = reinterpret_cast<WarpMem*>(s_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    WarpMem& M = all[wid];
    const float items = static_cast<float>(g.nwork);
    const float share = (static_cast<float>(st->candidates) * 64.f + kItemCost * items) /
                        static_cast<float>(gridDim.x * kWarps);
    const float heavy = kHeavy * share - kItemCost;
    if (lane == 0) M.evals = M.filtered = M.evals64 = M.bandc = 0;
    int64_t item = 0;  // the first of the grab
    bool own = false;  // the item in hand is this warp's (the first light one)
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) S.grab = atomicAdd(queue, 1ull);
        __syncthreads();
        item = static_cast<int64_t>(S.grab) * g.grab_n;
        if (item >= g.nwork) break;
        const int64_t b = g.work[item >> 6];
        if (static_cast<float>(g.cand_rng[2 * b + 1] - g.cand_rng[2 * b]) < heavy) {
            own = wid == 0;
            break;
        }
        for (int k = 0; k < g.grab_n && item + k < g.nwork; ++k)
            sub_brick<PREC, THIN, true>(g, item + k, M, S, all);
    }
    for (;;) {
        if (!own) {
            unsigned long long grab = 0;
            if (lane == 0) grab = atomicAdd(queue, 1ull);
            item = static_cast<int64_t>(__shfl_sync(kAll, grab, 0)) * g.grab_n;
        }
        own = false;
        if (item >= g.nwork) break;
        for (int k = 0; k < g.grab_n && item + k < g.nwork; ++k)
            sub_brick<PREC, THIN, false>(g, item + k, M, S, all);
    }
    if (lane == 0) {
        if (M.evals) atomicAdd(&st->evaluations, M.evals);
        if (M.filtered) atomicAdd(&st->filtered, M.filtered);
        if (M.evals64) atomicAdd(&st->fp64_evaluations, M.evals64);
        if (M.bandc) atomicAdd(&st->band_voxels, M.bandc);
    }
}

template <int PREC>
int near_grid() {
    int per = 0;
    CMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sdf_near<PREC, false>, 32 * kWarps,
                                                           kWarps * sizeof(WarpMem)));
    return device_sms() * (per > 0 ? per : 1);
}

}  // namespace

int sdf_near_grid(int precision) {
    return precision == kPrecMixed ? near_grid<kPrecMixed>() : near_grid<kPrecExact>();
}

void launch_sdf_near(int precision, bool thin, int grab, int probe, const MeshSeg* segs, int nseg,
                     const uint32_t* work, int64_t nwork, unsigned long long* queue,
                     const double* soup, const float4* tinfo, const float4* tinfo_lo,
                     const void* trec, const int64_t* cand_rng, const int* cand, const float4* cand_c,
                     float band_cells,
                     const uint8_t* occ, float* sdf32, double* sdf64, int* near_tri,
                     uint8_t* near_reg, float* errbound, Stats* stats, int grid, cudaStream_t st) {
    if (nwork == 0) return;
    if (grab != 1 && grab != 2 && grab != 4 && grab != 8) grab = 1;
    const int64_t need = (nwork + kWarps - 1) / kWarps;
    const unsigned blocks = static_cast<unsigned>(need < grid ? need : grid);
    const Args g{segs, nseg, work, nwork, grab, probe > 0 ? probe : INT_MAX, soup, tinfo, tinfo_lo,
                 static_cast<const TriRec*>(trec), cand_rng, cand, cand_c, band_cells,
                 {occ, sdf32, sdf64, near_tri, near_reg, errbound}};
    auto go = [&](auto kernel) {
        kernel<<<blocks, 32 * kWarps, kWarps * sizeof(WarpMem), st>>>(g, queue, stats);
    };
    if (precision == kPrecMixed) thin ? go(k_sdf_near<kPrecMixed, true>) : go(k_sdf_near<kPrecMixed, false>);
    else thin ? go(k_sdf_near<kPrecExact, true>) : go(k_sdf_near<kPrecExact, false>);
    CMG_LAUNCH();
}

}  // namespace cmg::gpu
