// Pairs of f32 in a 64-bit register and the packed operations on them (each half rounded as the scalar operation would).
#pragma once
#include <cstdint>

namespace infr {

typedef unsigned long long u64;
__device__ __forceinline__ u64 f2_pack(uint32_t lo, uint32_t hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ u64 f2_pack(float lo, float hi) { return f2_pack(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ u64 f2_dup(float v) { return f2_pack(v, v); }
__device__ __forceinline__ u64 f2_add(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 f2_mul(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 f2_fma(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

}  // namespace infr
