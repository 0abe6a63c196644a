// Per-format operations of the role-specialised kernel (one translation unit per storage format, so
// that they compile in parallel).
#pragma once

#include "step_launch.hpp"
#include "step_tiled.hpp"

namespace islbm {

struct RoleEntry {
    cudaError_t (*launch)(const StepLaunch &);
    size_t (*desc_bytes)();
    void (*fill)(const Tables<float> &, const StepConst &, const TiledConst &, Ctrl *, void *const macros[4], void *const buf[2],
                 const RoleMaps &, int ntiles, int nseg, void *out);
    cudaError_t (*launch_batch)(const void *descs, const int2 *items, int nitems, int grid, int macros_on, cudaStream_t);
    cudaError_t (*prepare)();
    size_t smem;
};
struct RoleTable {
    RoleEntry e[2][4];   // [LES][width 32, 64, 128, 256]
};
const RoleTable &roles_fp32();
const RoleTable &roles_fp16();
const RoleTable &roles_bf16();

}  // namespace islbm
