// Host-side launch descriptor shared by the ABI layer and the step kernels.
#pragma once

#include <cuda_runtime.h>

#include "../../include/islbm.h"
#include "step_common.cuh"

namespace islbm {

struct StepLaunch {
    int precision;             // islbm_precision
    const void *fo;            // 19*N populations, storage type
    void *fn;
    const void *tables;        // Tables<C> on the host (passed by value to the kernel)
    StepConst k;
    Ctrl *ctrl;                // device
    unsigned long long n;      // 1-based number of the step being computed
    unsigned seat_set;         // 0, 1, 0, ... over the step launches of the handle
    bool les, macros_on, mass;
    void *macros[4];           // rho, u, v, w (compute type) when macros_on
    const void *tiled;         // TiledConst for the tiled kernel
    const void *pmaps;         // paired kernel: the 4 tensor maps (CUtensorMap) of buffer fo, or null
    const void *chunk;         // ChunkConst for the chunk-marching kernel
    cudaStream_t stream;
};

// Programmatic dependent launch of consecutive step kernels: the next step's blocks may start, set up
// their barriers and tensor memory and then wait for the previous step's end and its memory
// (grid_dependency_wait) while that one's last blocks still run. A kernel launched this way touches no
// global memory before the wait but the seat words (claim_seat in step_roles.cuh: every block of the
// previous step has claimed its seat before it triggers). Populations are read with plain loads
// through pointers without __restrict__: the read-only path (__ldg, ld.global.nc) is for memory that
// nothing writes while the kernel is resident, and the previous step writes them until the wait
// ends. A read-only line cached by the step before that could be stale, and such a load may be
// moved above the wait. The tables, written at set-up only, may take that path.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

cudaError_t launch_step_gather(const StepLaunch &L);
cudaError_t launch_step_tiled(const StepLaunch &L);
bool tiled_supported(const StepConst &k, int precision);

}  // namespace islbm
