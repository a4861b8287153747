// int8 codes of the activation quantiser: `(v * id).round().clamp(-127.0, 127.0) as i8`
// (crates/infr-cpu/src/quant.rs:38, :71): round half away from zero; a NaN product gives 0 (what Rust's `as` makes of a
// NaN), an infinite one +-127.
#pragma once

namespace infr {

// x rounded half away from zero, |x| < 2^21, in the low byte of the result (two's complement); a NaN gives bits of its own.
// |x| + 0.5 and the sum with 2^23 are rounded towards zero: neither can reach an integer that the true sum does not reach, so what is
// left is floor(|x| + 0.5).  Four f32 additions and one integer instruction: conversions to integer and back run at a quarter of the f32
// rate, compares and selects at half of it, and a row is quantised by every CTA of a GEMV that takes f32 rows.
__device__ __forceinline__ uint32_t q8_round_bits(float x) {
    const float t = __fadd_rz(__fadd_rz(fabsf(x), 0.5f), 8388608.0f) - 8388608.0f;
    return __float_as_uint(copysignf(t, x) + 12582912.0f);
}

// The codes of four values in one word, the first in the low byte.  With a FINITE id, |v| <= amax and id = 1 / (amax / 127) a product
// stays below 127.5 in magnitude (two roundings of 2^-24 each), so rounding cannot leave [-127, 127].  An infinite id - a block whose
// largest magnitude is so small that amax / 127 has a reciprocal beyond the largest float - needs the clamp (both its comparisons are
// false for a NaN), and a NaN the zero: a branch of their own, which the empty asm keeps from becoming predicated instructions that every
// value pays for.  (Q4_K, 8 rows quantised inside the GEMV, 14336 -> 4096: 51.2 -> 47 us; by conversions, which the GEMV waits for, 48.1.  One Q2_0
// row 4096 -> 4096 4.0 -> 3.9.)
__device__ __forceinline__ uint32_t q8_codes4(const float4 v, float id) {
    float x[4] = {v.x * id, v.y * id, v.z * id, v.w * id};
    const float s = (x[0] + x[1]) + (x[2] + x[3]);  // (each is within +-127.5 or NaN where id is finite)
    if (!(id <= 3.0e38f) || s != s) {
        asm volatile("");
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = x[i] < -127.0f ? -127.0f : (x[i] > 127.0f ? 127.0f : x[i]);
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (x[i] != x[i]) x[i] = 0.f;
    }
    return __byte_perm(__byte_perm(q8_round_bits(x[0]), q8_round_bits(x[1]), 0x0040), __byte_perm(q8_round_bits(x[2]), q8_round_bits(x[3]), 0x0040), 0x5410);
}

// Sum of the four signed bytes of a word.
__device__ __forceinline__ int q8_sum4(uint32_t w) { return __dp4a((int)w, 0x01010101, 0); }

}  // namespace infr
