// Two packed floats as the f32x2 instructions take them, kept as one 64-bit value so that a pair stays in
// its aligned register pair (pairs of scalars cost moves around every packed instruction).
#pragma once

#include <cuda_runtime.h>

namespace opsblas {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 f2_pack(float x, float y)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ f32x2 f2_dup(float x) { return f2_pack(x, x); }
__device__ __forceinline__ void f2_unpack(f32x2 v, float& x, float& y)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ float f2_get(f32x2 v, int i)
{
    float x, y;
    f2_unpack(v, x, y);
    return i ? y : x;
}
// each half an IEEE fma
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// Each half rounded on its own. There is no packed sum here: the ptxas of CUDA 12.9 joins one with a packed
// product that feeds it into an fma, whatever roundings the two name.
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
}  // namespace opsblas
