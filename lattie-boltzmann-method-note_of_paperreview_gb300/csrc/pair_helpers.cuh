// Device helpers of the paired-node kernels: tensor-memory loads and stores of a thread's lane, node
// pairs in storage format, tensor-map copies.
#pragma once

#include <type_traits>

#include "pair_math.cuh"
#include "step_common.cuh"
#include "tile_helpers.cuh"

namespace islbm {
namespace {

__device__ __forceinline__ void tmem_st16(uint32_t ta, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(ta),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t ta, float a, float b, float c, float d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ta), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t ta, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(ta)
        : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t ta, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(ta)
                 : "memory");
}

// two stored values of adjacent nodes -> FP32 pair (the deviation formats give deviations)
template <class S> __device__ __forceinline__ V2 ld2v(const S *p);
template <> __device__ __forceinline__ V2 ld2v<float>(const float *p) { return V2(*(const float2 *)p); }
template <> __device__ __forceinline__ V2 ld2v<__half>(const __half *p) { return V2(__half22float2(*(const __half2 *)p)); }
template <> __device__ __forceinline__ V2 ld2v<__nv_bfloat16>(const __nv_bfloat16 *p) {
    return V2(__bfloat1622float2(*(const __nv_bfloat162 *)p));
}
// full values of a node pair from global memory (plain loads: see grid_dependency_wait)
template <class S> __device__ __forceinline__ V2 ld2g(const S *p, int q) {
    V2 v;
    if constexpr (std::is_same<S, float>::value) v = V2(*(const float2 *)p);
    else if constexpr (std::is_same<S, __half>::value) {
        const unsigned r = *(const unsigned *)p;
        v = V2(__half22float2(*(const __half2 *)&r));
    } else {
        const unsigned r = *(const unsigned *)p;
        v = V2(__bfloat1622float2(*(const __nv_bfloat162 *)&r));
    }
    if constexpr (Storage<S>::dev) v = v + V2((float)dev_ref(q));
    return v;
}
// store a node pair (full values; the deviation formats store f - ref)
template <class S> __device__ __forceinline__ void st2(S *p, V2 v, int q) {
    if constexpr (std::is_same<S, float>::value) *(float2 *)p = v.v;
    else {
        const V2 d = v - V2((float)dev_ref(q));
        if constexpr (std::is_same<S, __half>::value) *(__half2 *)p = __float22half2_rn(d.v);
        else *(__nv_bfloat162 *)p = __float22bfloat162_rn(d.v);
    }
}

// Tensor copy of one box (x, y, z, q) of a population buffer: the box lands in shared memory as
// [q][rows][NX], the layout of the front and stage buffers.
__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *map, int x, int y, int z, int q, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(smem_u32(dst)), "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(q), "r"(smem_u32(bar))
                 : "memory");
}

}  // namespace
}  // namespace islbm
