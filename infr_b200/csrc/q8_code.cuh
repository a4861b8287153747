// One int8 code of the activation quantiser: `(v * id).round().clamp(-127.0, 127.0) as i8`
// (crates/infr-cpu/src/quant.rs:38, :71): round half away from zero; a NaN product gives 0 (what Rust's `as` makes of a
// NaN), an infinite one +-127.
#pragma once

namespace infr {

// x rounded half away from zero, |x| < 2^21, as the low bits of the result (two's complement, 0x4B400000 = 0); a NaN gives low bits of its
// own.  |x| + 0.5 and the sum with 2^23 are rounded towards zero: neither can reach an integer that the true sum does not reach, so what is
// left is floor(|x| + 0.5).  Four f32 additions and one integer instruction: conversions to integer and back run at a quarter of the f32
// rate, compares and selects at half of it, and a row is quantised by every CTA of a GEMV that takes f32 rows.
__device__ __forceinline__ uint32_t q8_round_bits(float x) {
    const float t = __fadd_rz(__fadd_rz(fabsf(x), 0.5f), 8388608.0f) - 8388608.0f;
    return __float_as_uint(copysignf(t, x) + 12582912.0f);
}
__device__ __forceinline__ int q8_round(float x) { return x == x ? (int)(q8_round_bits(x) - 0x4B400000u) : 0; }

__device__ __forceinline__ int q8_round_code(float v, float id) {
    float x = v * id;
    x = x < -127.0f ? -127.0f : (x > 127.0f ? 127.0f : x);  // both comparisons are false for a NaN: it passes through
    return q8_round(x);
}

// The same without the clamp, for a FINITE id: with |v| <= amax and id = 1 / (amax / 127) the product stays below
// 127.5 in magnitude (two roundings of 2^-24 each), so rounding cannot leave [-127, 127].  (An infinite id - a block
// whose largest magnitude is so small that amax / 127 has a reciprocal beyond the largest float - needs the clamp.)
__device__ __forceinline__ int q8_round_code_inrange(float v, float id) { return q8_round(v * id); }

// Four codes in one word, the first in the low byte (the codes are within [-127, 127]: the saturation never acts).
__device__ __forceinline__ uint32_t q8_pack4(int q0, int q1, int q2, int q3) {
    uint32_t hi, w;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q3), "r"(q2));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q1), "r"(q0), "r"(hi));
    return w;
}

// The codes of four values in one word, the first in the low byte.
__device__ __forceinline__ uint32_t q8_codes4(const float4 v, float id) {
    float x[4] = {v.x * id, v.y * id, v.z * id, v.w * id};
    if (!(id <= 3.0e38f)) {  // an infinite id (see q8_round_code)
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = x[i] < -127.0f ? -127.0f : (x[i] > 127.0f ? 127.0f : x[i]);
    }
    uint32_t w = __byte_perm(__byte_perm(q8_round_bits(x[0]), q8_round_bits(x[1]), 0x0040), __byte_perm(q8_round_bits(x[2]), q8_round_bits(x[3]), 0x0040), 0x5410);
    const float s = (x[0] + x[1]) + (x[2] + x[3]);  // (each is within +-127.5 or NaN)
    if (s != s) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (x[i] != x[i]) w &= ~(0xFFu << (8 * i));
    }
    return w;
}

// Sum of the four signed bytes of a word.
__device__ __forceinline__ int q8_sum4(uint32_t w) { return __dp4a((int)w, 0x01010101, 0); }

}  // namespace infr
