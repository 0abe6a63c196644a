// Launch constants of the chunk-marching step kernel (step_chunk.cu), computed once per solve.
#pragma once

#include <stddef.h>

#include <cuda_runtime.h>

#include "step_common.cuh"
#include "step_launch.hpp"

namespace islbm {

struct ChunkConst {
    int W, H;                  // columns and rows of a tile (W*H <= 32 lanes)
    int tiles_x, tiles_y;
    int segs;                  // wall-normal segments per column
    int grid;                  // persistent CTAs
    unsigned inv_hw, inv_wh;   // 2^32/(H*(W + 6)) (FP32: H + 6) and 2^32/(W + 6), rounded up: exact quotients by __umulhi
    size_t smem_bytes;
    double wx0[7], wx2[7], wy0[7], wy2[7];   // uniform-spacing Lagrange weights
};

// byte offsets into a population array are 32-bit in the kernel; larger grids keep the gather kernel
bool chunk_supported(const StepConst &k, int precision);
// tile, segments and grid for a solve on the current device (which must be the solve's)
cudaError_t make_chunk_const(const StepConst &k, int precision, bool les, const double *wx0, const double *wx2,
                             const double *wy0, const double *wy2, int num_sms, ChunkConst *out);
cudaError_t launch_step_chunk(const StepLaunch &L);

}  // namespace islbm
