// f32x2.cuh -- two floats per instruction.  sm_103a's packed single-precision
// add, multiply and multiply-add take one issue slot for two results (and the
// cycles of two), so kernels bound by instruction issue work on pairs of
// x-adjacent voxels.  Every half is rounded as the scalar instruction rounds.
#pragma once

#include <cuda_runtime.h>

namespace m16 {

typedef unsigned long long f2;   // low word: the first float

__device__ __forceinline__ f2 pack2(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 both2(float v) { return pack2(v, v); }
__device__ __forceinline__ float lo2(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, both2(-1.f), a); }

}  // namespace m16
