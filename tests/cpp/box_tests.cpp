// The distance kernels' pruning tests (csrc/cmg_sdf.cuh) compiled for the host, so that their
// margins can be tried without a GPU: the header itself, with the few intrinsics it names.
// The approximate square root gives its lowest value.
#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>

inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __ddiv_rn(double a, double b) { return a / b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __saturatef(float a) { return a > 0.f ? (a < 1.f ? a : 1.f) : 0.f; }
inline float __double2float_rn(double a) { return static_cast<float>(a); }
inline long long __double_as_longlong(double a) {
    long long b;
    std::memcpy(&b, &a, 8);
    return b;
}
template <typename T>
T __ldg(const T* p) { return *p; }
template <typename T>
T __shfl_xor_sync(unsigned, T v, int) { return v; }
template <typename T>
T min(T a, T b) { return a < b ? a : b; }

#ifndef __noinline__
#define __noinline__
#endif
#define asm(...) y = std::sqrt(x) * (1.f - 1.2e-7f)
#include "cmg_sdf.cuh"
#undef asm

using namespace cmg::gpu::sdf;

namespace {
// b: q (3), h (3), r, eps, pos
BoxTest box(const float* b) { return box_test(b[0], b[1], b[2], b[3], b[4], b[5], b[6], b[7], b[8]); }
}  // namespace

extern "C" {
float normal_error() { return kRecNormalErr; }
int ball(const float* b, const float* c, float w) { return box_ball(box(b), c[0], c[1], c[2], w, b[8]); }
int disc(const float* b, const float* c, float w, const float* n, float nerr) {
    return box_disc(box(b), c[0], c[1], c[2], w, make_float4(n[0], n[1], n[2], nerr));
}
int cell(float d2, float pn, float b, float w) { return cell_disc(d2, pn, b, w); }
}
