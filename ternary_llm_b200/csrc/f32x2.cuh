// Two FP32 numbers in a 64-bit register pair, multiplied and added by one instruction.
#pragma once
#include <cstdint>

namespace tllm {

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pair_f32(uint32_t lo, uint32_t hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ f32x2 pair_f32(float lo, float hi) { return pair_f32(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ float2 split_f32(f32x2 v)
{
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}
__device__ __forceinline__ void fma_pair(f32x2& acc, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ f32x2 mul_pair(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add_pair(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float sum_pair(f32x2 v)
{
    const float2 f = split_f32(v);
    return f.x + f.y;
}

}  // namespace tllm
