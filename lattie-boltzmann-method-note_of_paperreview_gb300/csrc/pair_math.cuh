// Packed arithmetic on node pairs: every FP32 operation of the paired-node step kernel works
// on (node x, node x + 1) at once through the FP32x2 instructions of sm_100+ (add, mul and fma
// on a float2 in one instruction). A product followed by an addition or subtraction is
// contracted into one fused multiply-add, as the compiler does for scalar FP32 code.
#pragma once

#include <cuda_runtime.h>

#include "collide.cuh"

namespace islbm {

struct V2 {
    float2 v;
    __device__ __forceinline__ V2() {}
    __device__ __forceinline__ V2(float2 a) : v(a) {}
    __device__ __forceinline__ V2(float a, float b) : v(make_float2(a, b)) {}
    // broadcast constants (the generated MRT code writes T(c))
    __device__ __forceinline__ explicit V2(double c) : v(make_float2((float)c, (float)c)) {}
    __device__ __forceinline__ explicit V2(float c) : v(make_float2(c, c)) {}
    __device__ __forceinline__ explicit V2(int c) : v(make_float2((float)c, (float)c)) {}
};

__device__ __forceinline__ V2 vneg(V2 a) { return V2(-a.v.x, -a.v.y); }
__device__ __forceinline__ V2 vadd(V2 a, V2 b) { return V2(__fadd2_rn(a.v, b.v)); }
__device__ __forceinline__ V2 vsub(V2 a, V2 b) { return V2(__fadd2_rn(a.v, vneg(b).v)); }
__device__ __forceinline__ V2 vmul(V2 a, V2 b) { return V2(__fmul2_rn(a.v, b.v)); }
__device__ __forceinline__ V2 vfma(V2 a, V2 b, V2 c) { return V2(__ffma2_rn(a.v, b.v, c.v)); }

// a product not yet rounded: consumed by + or - as one fused multiply-add
struct V2M {
    V2 a, b;
    __device__ __forceinline__ operator V2() const { return vmul(a, b); }
};
__device__ __forceinline__ V2M operator*(V2 a, V2 b) { return V2M{a, b}; }
__device__ __forceinline__ V2M operator*(V2M m, V2 c) { return V2M{vmul(m.a, m.b), c}; }
__device__ __forceinline__ V2M operator*(V2 c, V2M m) { return V2M{c, vmul(m.a, m.b)}; }
__device__ __forceinline__ V2M operator*(V2M m, V2M n) { return V2M{vmul(m.a, m.b), vmul(n.a, n.b)}; }
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return vadd(a, b); }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return vsub(a, b); }
__device__ __forceinline__ V2 operator-(V2 a) { return vneg(a); }
__device__ __forceinline__ V2 operator+(V2M m, V2 c) { return vfma(m.a, m.b, c); }
__device__ __forceinline__ V2 operator+(V2 c, V2M m) { return vfma(m.a, m.b, c); }
__device__ __forceinline__ V2 operator+(V2M m, V2M n) { return vfma(m.a, m.b, vmul(n.a, n.b)); }
__device__ __forceinline__ V2 operator-(V2 c, V2M m) { return vfma(vneg(m.a), m.b, c); }
__device__ __forceinline__ V2 operator-(V2M m, V2 c) { return vfma(m.a, m.b, vneg(c)); }
__device__ __forceinline__ V2 operator-(V2M m, V2M n) { return vfma(m.a, m.b, vneg(vmul(n.a, n.b))); }
__device__ __forceinline__ V2M operator-(V2M m) { return V2M{vneg(m.a), m.b}; }
__device__ __forceinline__ V2 &operator+=(V2 &a, V2 b) { a = vadd(a, b); return a; }
__device__ __forceinline__ V2 &operator-=(V2 &a, V2 b) { a = vsub(a, b); return a; }
__device__ __forceinline__ V2 &operator+=(V2 &a, V2M m) { a = vfma(m.a, m.b, a); return a; }
__device__ __forceinline__ V2 &operator-=(V2 &a, V2M m) { a = vfma(vneg(m.a), m.b, a); return a; }

// per-lane reciprocal and square root (no packed forms)
__device__ __forceinline__ V2 c_rcp(V2 a) { return V2(c_rcp(a.v.x), c_rcp(a.v.y)); }
__device__ __forceinline__ V2 c_sqrt(V2 a) { return V2(c_sqrt(a.v.x), c_sqrt(a.v.y)); }

}  // namespace islbm
