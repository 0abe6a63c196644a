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
    size_t smem_bytes;
    double wx0[7], wx2[7], wy0[7], wy2[7];   // uniform-spacing Lagrange weights
};

// tile, segments and grid for a solve on the current device (which must be the solve's)
cudaError_t make_chunk_const(const StepConst &k, int precision, bool les, const double *wx0, const double *wx2,
                             const double *wy0, const double *wy2, int num_sms, ChunkConst *out);
cudaError_t launch_step_chunk(const StepLaunch &L);

}  // namespace islbm
