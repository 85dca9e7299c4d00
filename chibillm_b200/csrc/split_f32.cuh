// 32-bit numbers two at a time, and as three bfloat16 numbers for the tensor cores.
//
// A 32-bit number is the sum of three bfloat16 numbers (its leading 8 bits, the next 8 of what is left, and the last 8;
// each rounded to nearest: Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence datatype for
// higher-precision computations", 2019), so a product of two is the sum of nine exact products of 8 by 8 bits.  The users of
// this file leave the three smallest out (each at most 2^-25 of the whole, together at most 2^-24) and make the other six with
// 32-bit accumulators.
//
// Numbers are split times 2^16, so that the last parts of small ones are no smaller than a bfloat16 can be.  What is no number, or
// too large (from 2^112 on), has an infinite part and a rest that is no number.
#pragma once
#include "common.cuh"

namespace chibi {

__device__ __forceinline__ uint64_t pair_of(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 halves_of(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t pair_fma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pair_add(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t pair_mul(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

constexpr uint64_t PAIR_ONES = 0x3f8000003f800000ull, PAIR_MINUS_ONES = 0xbf800000bf800000ull;
constexpr uint64_t SPLIT_UP = 0x4780000047800000ull;         // 2^16 twice
constexpr float SPLIT_DOWN = 0x1p-32f;                       // for a product of two numbers that were split

// Two numbers as bfloat16, the first in the lower half.
__device__ __forceinline__ uint32_t bf16_pair(uint64_t v)
{
    const float2 h = halves_of(v);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(h.y), "f"(h.x));
    return r;
}
// What is left of two numbers without their bfloat16 parts (exact).
__device__ __forceinline__ uint64_t without_bf16_pair(uint64_t v, uint32_t pair)
{
    return pair_fma(pair_of(__uint_as_float(pair << 16), __uint_as_float(pair & 0xffff0000u)), PAIR_MINUS_ONES, v);
}
// The three parts of four numbers, two to a word.  Returns what the last parts were before they were rounded, added up: no
// number where one of the four has no parts.
__device__ __forceinline__ uint64_t split_parts(float4 v, uint32_t (&parts)[3][2])
{
    uint64_t x = pair_mul(pair_of(v.x, v.y), SPLIT_UP), y = pair_mul(pair_of(v.z, v.w), SPLIT_UP);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        parts[i][0] = bf16_pair(x);
        parts[i][1] = bf16_pair(y);
        if (i < 2) {
            x = without_bf16_pair(x, parts[i][0]);
            y = without_bf16_pair(y, parts[i][1]);
        }
    }
    return pair_add(x, y);
}
// The same, written to shared memory `plane` bytes apart.
__device__ __forceinline__ uint64_t split_to_shared(float4 v, uint32_t at, uint32_t plane)
{
    uint32_t parts[3][2];
    const uint64_t last = split_parts(v, parts);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + i * plane), "r"(parts[i][0]), "r"(parts[i][1]) : "memory");
    return last;
}
// Whether one of two numbers is none or infinite.
__device__ __forceinline__ bool pair_is_none(uint64_t v)
{
    const float2 h = halves_of(v);
    return !(fabsf(h.x + h.y) < INFINITY);
}

} // namespace chibi
