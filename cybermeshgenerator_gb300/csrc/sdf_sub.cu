// sdf_sub.cu — plain FP64 distance per cell (CMG_PREC_FP64_PLAIN), evaluated in 4^3
// sub-bricks of the 16^3 candidate bricks: every candidate in FP64, no FP32 pass (the
// same results as sdf_near.cu's exact path, for comparison).
//
// One 64-thread CTA per 4^3 sub-brick (a persistent kernel over an LPT-ordered queue of
// sub-bricks):
//   1. probe: an upper bound U on the distance from the sub-brick centre c to the
//      surface (FP32 point-triangle distance with its error bound, over the brick
//      list, each thread skipping triangles whose bounding sphere is beyond its
//      own bound so far);
//   2. filter: the brick list is compacted in shared memory to the triangles whose
//      bounding sphere and plane can reach U + 2 r (r the sub-brick radius) — in rounds of
//      at most kCap entries;
//   3. cells, one per thread: bounding-sphere and plane tests per listed triangle, and
//      the distance (Ericson in the reference order) only when some lane of the warp
//      needs it.
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

constexpr int kSubThreads = 64;  // one cell per thread
constexpr int kCap = 256;        // filtered candidates per round in shared memory
constexpr int kBatch = 4;        // candidates per thread per probe/filter step (loads in flight)
static_assert(kCap >= kBatch * kSubThreads, "a round must hold one filter step");

// MINB: resident CTAs per SM the registers are budgeted for (12: 80 registers; 16: 64).
// grab: consecutive sub-bricks taken from the queue at once (a divisor of 64: they share
// one brick list).
template <int MINB>
__global__ void __launch_bounds__(kSubThreads, MINB)
k_sdf_sub(const MeshSeg* __restrict__ segs, int nseg, const uint32_t* __restrict__ work,
          int64_t nwork, int grab_n, unsigned long long* __restrict__ queue,
          const double* __restrict__ soup,
          const float4* __restrict__ tinfo, const float4* __restrict__ tinfo_lo,
          const TriRec* __restrict__ trec, const float4* __restrict__ tnorm,
          const int64_t* __restrict__ cand_rng,
          const int* __restrict__ cand, Out o, Stats* __restrict__ st) {
    __shared__ float4 s_c[kCap];  // centroid relative to the sub-brick centre, radius
    // unit normal and plane offset n . centroid, and a bound on the error of the plane
    // distances computed from them
    __shared__ float4 s_nrm[kCap];
    __shared__ float s_pe[kCap];
    __shared__ int s_t[kCap];
    __shared__ int s_n;
    __shared__ long long s_item;
    __shared__ unsigned long long s_red[kSubThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long evals = 0;

    for (;;) {
        if (tid == 0) s_item = static_cast<long long>(atomicAdd(queue, 1ull));
        __syncthreads();
        const int64_t grab = s_item;
        __syncthreads();
        if (grab * grab_n >= nwork) break;
      for (int gi = 0; gi < grab_n; ++gi) {
        const int64_t item = grab * grab_n + gi;
        if (item >= nwork) break;
        const int64_t gb = work[item >> 6];  // the bricks in order, 64 sub-bricks each
        const int sub = static_cast<int>(item & 63);
        const MeshSeg& s = segs[find_seg<&MeshSeg::brick_begin>(segs, nseg, gb)];
        const GridDesc g = s.g;
        const SubGeo q = sub_geo(s, gb - s.brick_begin, sub);
        if (q.empty) continue;
        // sub-brick centre relative to the grid corner, as an FP32 hi + lo pair
        const double ckx = 0.5 * (q.x0 + q.x1) * g.h, cky = 0.5 * (q.y0 + q.y1) * g.h,
                     ckz = 0.5 * (q.z0 + q.z1) * g.h;
        float chx, clx, chy, cly, chz, clz;
        split2(ckx, chx, clx);
        split2(cky, chy, cly);
        split2(ckz, chz, clz);
        const double hx = 0.5 * (q.x1 - q.x0 - 1) * g.h, hy = 0.5 * (q.y1 - q.y0 - 1) * g.h,
                     hz = 0.5 * (q.z1 - q.z0 - 1) * g.h;
        const float r4 = __double2float_ru(sqrt(hx * hx + hy * hy + hz * hz) * (1.0 + 1e-9));
        // this thread's cell
        const int x = q.x0 + (tid & 3), y = q.y0 + ((tid >> 2) & 3), z = q.z0 + (tid >> 4);
        const bool valid = x < q.x1 && y < q.y1 && z < q.z1 && z >= g.z0 && z < g.z1;
        const float px = static_cast<float>((x + 0.5) * g.h - ckx);
        const float py = static_cast<float>((y + 0.5) * g.h - cky);
        const float pz = static_cast<float>((z + 0.5) * g.h - ckz);
        const int64_t c0 = cand_rng[2 * gb], c1 = cand_rng[2 * gb + 1];

        // ---- 1. probe: upper bound on the distance from the centre to the surface,
        //         and the triangle that gives it (the seed of every cell below)
        float tb = FLT_MAX;
        int tseed = INT_MAX;
        for (int64_t k0 = c0 + tid; k0 < c1; k0 += kBatch * kSubThreads) {
            // loads of kBatch candidates in flight before any of them is used
            int tt[kBatch];
            float4 hh[kBatch], ll[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                const int64_t k = k0 + i * kSubThreads;
                tt[i] = k < c1 ? cand[k] : -1;
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i)
                if (tt[i] >= 0) { hh[i] = tinfo[tt[i]]; ll[i] = tinfo_lo[tt[i]]; }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (tt[i] < 0) continue;
                const int t = tt[i];
                const float4 hi = hh[i], lo = ll[i];
                const float rx = (hi.x - chx) + (lo.x - clx);
                const float ry = (hi.y - chy) + (lo.y - cly);
                const float rz = (hi.z - chz) + (lo.z - clz);
                const float dc = sqrtf(rx * rx + ry * ry + rz * rz);
                const float sb = (dc + hi.w) * (1.f + 8.f * kU32);  // bounding-sphere bound
                if (sb < tb) { tb = sb; tseed = t; }
                if (dc - hi.w < tb) {
                    TriRec r;
                    load_rec(trec, t, r);
                    const float d = sqrtf(dist_rec_val(r, -rx, -ry, -rz));
                    const float ub = d * (1.f + 32.f * kU32) + 32.f * kU32 * (dc + 2.f * hi.w);
                    if (ub < tb || (ub == tb && t < tseed)) { tb = ub; tseed = t; }
                }
            }
        }
        // block argmin of (bound, triangle): bound bits first, then the id
        unsigned long long key =
            (static_cast<unsigned long long>(__float_as_uint(tb)) << 32) | static_cast<unsigned>(tseed);
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
            const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, sh);
            key = k2 < key ? k2 : key;
        }
        if (lane == 0) s_red[warp] = key;
        __syncthreads();
        unsigned long long kmin = s_red[0];
#pragma unroll
        for (int i = 1; i < kSubThreads / 32; ++i) kmin = s_red[i] < kmin ? s_red[i] : kmin;
        const float U = __uint_as_float(static_cast<unsigned>(kmin >> 32));
        const int seed = static_cast<int>(static_cast<unsigned>(kmin & 0xffffffffull));
        // a triangle can be nearest to a cell only if its sphere reaches U + 2 r
        const float limf = (U + 2.f * r4) * (1.f + 32.f * kU32) + 32.f * kU32 * (U + r4);

        // ---- 2+3. rounds: filter into shared memory, then evaluate the cells
        float bestd = FLT_MAX;
        double best64 = DBL_MAX;
        int bt = INT_MAX, br = 0;
        const d3 P{cell_center(g.corner[0], x, g.h), cell_center(g.corner[1], y, g.h),
                   cell_center(g.corner[2], z, g.h)};
        auto evaluate = [&](int t) {
            d3 a, b, c;
            load_soup(soup, t, a, b, c);
            if (valid) {
                int reg;
                const double d2 = ericson(P, a, b, c, &reg);
                ++evals;
                if (d2 < best64 || (d2 == best64 && t < bt)) {
                    best64 = d2;
                    bt = t;
                    br = reg;
                    bestd = __double2float_ru(sqrt(d2)) * (1.f + 8.f * kU32);
                }
            }
        };
        // the centre's nearest triangle: a tight start for every cell's bound
        if (seed != INT_MAX) evaluate(seed);
        int64_t cursor = c0;
        while (cursor < c1) {
            if (tid == 0) s_n = 0;
            __syncthreads();
            int n = 0;
            while (cursor < c1 && n <= kCap - kBatch * kSubThreads) {
                int tt[kBatch];
                float4 hh[kBatch], ll[kBatch];
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    const int64_t k = cursor + tid + i * kSubThreads;
                    tt[i] = k < c1 ? cand[k] : -1;
                }
#pragma unroll
                for (int i = 0; i < kBatch; ++i)
                    if (tt[i] >= 0) { hh[i] = tinfo[tt[i]]; ll[i] = tinfo_lo[tt[i]]; }
#pragma unroll
                for (int i = 0; i < kBatch; ++i) {
                    bool take = false;
                    float4 e = make_float4(0.f, 0.f, 0.f, 0.f), nv = e;
                    float pe = 0.f;
                    const int t = tt[i];
                    if (t >= 0) {
                        e.x = (hh[i].x - chx) + (ll[i].x - clx);
                        e.y = (hh[i].y - chy) + (ll[i].y - cly);
                        e.z = (hh[i].z - chz) + (ll[i].z - clz);
                        e.w = hh[i].w;
                        const float dc = sqrtf(e.x * e.x + e.y * e.y + e.z * e.z);
                        // the plane's distance from a cell is at most its distance from the
                        // triangle, so a triangle whose plane stays beyond every cell's
                        // reach (U + r from the centre) cannot be nearest to any of them. pe
                        // bounds the plane distances' error at any cell of the sub-brick
                        // (normal error n.w; rounding of the FP32 centroid, cell offsets and
                        // dot products)
                        take = dc - e.w <= limf;
                        if (take) {
                            nv = tnorm[t];
                            pe = (nv.w + 12.f * kU32) * (dc + r4) * 1.1f + 1e-30f;
                            nv.w = fmaf(nv.x, e.x, fmaf(nv.y, e.y, nv.z * e.z));
                            take = fabsf(nv.w) - pe <= limf;
                        }
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, take);
                    int base = 0;
                    if (lane == 0 && m) base = atomicAdd(&s_n, __popc(m));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (take) {
                        const int pos = base + __popc(m & ((1u << lane) - 1u));
                        s_c[pos] = e;
                        s_nrm[pos] = nv;
                        s_pe[pos] = pe;
                        s_t[pos] = t;
                    }
                }
                cursor += kBatch * kSubThreads;
                __syncthreads();
                n = s_n;
            }
            if (tid == 0 && n) atomicAdd(&st->filtered, static_cast<unsigned long long>(n));
            for (int j = 0; j < n; ++j) {
                const float4 e = s_c[j];
                const float dx = px - e.x, dy = py - e.y, dz = pz - e.z;
                const float lim = (bestd + e.w) * (1.f + 16.f * kU32) + 16.f * kU32 * r4;
                bool need = valid && dx * dx + dy * dy + dz * dz <= lim * lim;
                if (!__any_sync(0xffffffffu, need)) continue;
                // and the plane: its distance from the cell bounds the triangle's below
                const float4 nv = s_nrm[j];
                const float pd = fabsf(fmaf(nv.x, px, fmaf(nv.y, py, fmaf(nv.z, pz, -nv.w))));
                need = need && pd - s_pe[j] <= bestd * (1.f + 16.f * kU32) + 16.f * kU32 * r4;
                if (!__any_sync(0xffffffffu, need)) continue;
                evaluate(s_t[j]);
            }
            __syncthreads();
        }
        if (valid)
            write_cell(o, s.vox_begin + (static_cast<int64_t>(z - g.z0) * g.ny + y) * g.nx + x,
                       __dsqrt_rn(best64), bt, br);
        __syncthreads();
      }
    }
    const long long ev = warp_sum(static_cast<long long>(evals));
    if (lane == 0 && ev) {
        atomicAdd(&st->evaluations, static_cast<unsigned long long>(ev));
        atomicAdd(&st->fp64_evaluations, static_cast<unsigned long long>(ev));
    }
}

}  // namespace

// Resident CTAs per SM targeted by the evaluation kernel: 16 when asked for, else 12.
int sdf_sub_minb(int ctas) { return ctas == 16 ? 16 : 12; }

int sdf_sub_grid(int ctas) {
    int per = 0;
    if (sdf_sub_minb(ctas) == 16)
        CMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sdf_sub<16>, kSubThreads, 0));
    else CMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sdf_sub<12>, kSubThreads, 0));
    return device_sms() * (per > 0 ? per : 1);
}

void launch_sdf_sub(int grab, int ctas, const MeshSeg* segs, int nseg, const uint32_t* work,
                    int64_t nwork, unsigned long long* queue, const double* soup,
                    const float4* tinfo, const float4* tinfo_lo, const void* trec,
                    const float4* tnorm, const int64_t* cand_rng, const int* cand,
                    const uint8_t* occ, float* sdf32, double* sdf64, int* near_tri,
                    uint8_t* near_reg, Stats* stats, int grid, cudaStream_t st) {
    if (nwork == 0) return;
    Out o{occ, sdf32, sdf64, near_tri, near_reg, nullptr};
    const TriRec* r = static_cast<const TriRec*>(trec);
    if (grab != 1 && grab != 2 && grab != 4 && grab != 8) grab = 1;
    auto go = [&](auto kernel) {
        kernel<<<grid, kSubThreads, 0, st>>>(segs, nseg, work, nwork, grab, queue, soup, tinfo,
                                            tinfo_lo, r, tnorm, cand_rng, cand, o, stats);
    };
    sdf_sub_minb(ctas) == 16 ? go(k_sdf_sub<16>) : go(k_sdf_sub<12>);
    CMG_LAUNCH();
}

}  // namespace cmg::gpu
