// One activation row against block-quantized matrices (Q4_K, Q6_K, Q2_0): the matvec of a decoded token.
//
// Arithmetic of crates/infr-cpu/src/kernels.rs:151-184 (Q4_K), :487-526 (Q6_K), :5641-5668 (Q2_0): the products of every sub-block
// (32, 16, 32 elements) are exact int32 sums of 8-bit codes, sub-block scales are applied in int32, block scales in f32.
//
// `mma.sync.m16n8k32.u8.s8` multiplies 16 weight rows by 8 columns, and there is one activation row.  The columns are the SUB-BLOCKS:
// column s of B holds the codes of sub-block s and zero in the K slots of all others, so that one accumulator collects the sums of eight
// sub-blocks side by side, spread over all lanes: a lane scales 2 rows x 2 sub-blocks, where a column per activation row had one lane
// in four scale 2 rows x 8.
// The codes of B that a lane needs are its own 8 bytes of a block: read straight into registers, or quantised there from f32 rows (the
// lane that quantises an element is the lane that multiplies it), without a staging copy that the warps of a CTA wait for.
//
// The warps of a CTA split K; a warp's units (Q4_K 256 elements, Q6_K and Q2_0 512) come by tiled TMA, 16 rows a box, through a ring of its
// own.  (More slots a warp: the warps drift apart, neighbouring 144-byte pieces of a weight row are fetched at different times, and
// 4096 -> 128256 takes 55 us with three slots and 68 with four instead of 49 with two.)
// Q4_K and Q6_K: every block's term meets the others in shared memory, a few tiles at a time, and the terms of a row are added in the order
// that row_group says: that of the kernels for two rows and more, had they one.  (A sum in another order differs in a last bit here and
// there, and 32 layers that code their activations in 8 bits carry that on to 0.01 .. 0.03 of a model's result.)  Q2_0: chains of blocks in the
// order of the byte-dot kernel, for the same reason (kQ2Chains).
// All waits are bounded; an expired one records a status word for the host.
// Measured (us a call in a chain of calls on cold weights; before = the columns-are-rows kernels, or the byte-dot kernel for Q2_0; codes / f32
// rows): Q4_K 4096 -> 4096 3.5 / 4.4 -> 3.6 / 3.9, 4096 -> 14336 7.5 / 9.4 -> 7.8 / 8.0, 14336 -> 4096 8.5 / 11.5 -> 8.0 / 9.9;  Q6_K
// 4096 -> 4096 5.3 / 6.8 -> 4.5 / 4.5, 4096 -> 14336 13.1 / 15.1 -> 10.1 / 10.1, 4096 -> 128256 79 -> 65;  Q2_0 4096 -> 4096 4.5 / 5.6 -> 3.1 / 4.0,
// 14336 -> 4096 8.4 / 10.4 -> 7.0 / 9.6, 4096 -> 128256 54 -> 33.  Between other launches (the decode step of an 8B model) the Q4_K shapes gain
// more: their CTAs leave room for the launch before.  Long rows of few tiles, codes of more than 16 blocks and rows whose terms leave no room are
// faster there still and go there (row_first in gemv_mma.cu, the lines in launch_gemv_q6_mma and CudaBackend::linear).
// What bounds it: small matrices the chain from one launch to the next (1 us) and one round trip to L2 for the activations (0.3 us);
// large ones memory (4096 -> 128256 at 0.92 of the measured copy rate, Q6_K 1.0); Q2_0 the integer pipe (64 masks a unit, half rate).
#include <cuda.h>

#include <atomic>
#include <cstring>

#include "gemv_common.cuh"
#include "q8_code.cuh"

namespace infr {
namespace {

constexpr int kRowTile = 16;
constexpr int kRowSlots = 3;   // ring slots of a warp, at most
constexpr uint32_t kRowSpin = 1u << 22;

// kPart: tiles whose sums wait for one barrier; kTerm: floats of a block's term (Q4_K: d * sum - dmin * min sum, times the row's scale when
// it is added; Q6_K: both factors).
// kUnit elements of a row are one box of 16 rows x kPitch bytes.  A Q6_K unit (two blocks, 420 bytes) starts on a multiple of 4: its box
// starts at the 16-byte boundary below.  Pitches of 36 and 108 words put the eight rows of a read on distinct banks.
template <int DT>
struct RowFmt;
template <>
struct RowFmt<DT_Q4K> {
    static constexpr int kUnit = 256, kPitch = 144, kActBytes = 256 + 32, kWarps = 16, kPart = 4, kTerm = 1;
};
template <>
struct RowFmt<DT_Q6K> {
    static constexpr int kUnit = 512, kPitch = 432, kActBytes = 512 + 64 + 16, kWarps = 8, kPart = 2, kTerm = 2;
};
template <>
struct RowFmt<DT_Q2_0> {
    static constexpr int kUnit = 512, kPitch = 144, kActBytes = 512 + 128, kWarps = 16, kPart = 1, kTerm = 2;
};
// Q2_0: a result is the sum of 32 chains (block b of the row is added to chain b mod 32, in order) along a fixed tree, the order of the byte-dot
// kernel (gemv_stream.cu), whose bits a model keeps.  A unit's eight blocks belong to eight chains, those of unit u to eight of class u mod 4.
// Short rows: four warps, each takes the units of a class and its lanes keep the chains; long rows, which four warps are too few for: up to 16,
// every block's integer sums and scale meet in shared memory and a warp a row adds them.
constexpr int kQ2ChainWarps = 4;
constexpr int kQ2Stride = 24, kQ2Chains = 8 * kQ2Stride;  // floats between a tile's chains of one class (16 rows, padded: no bank conflicts)
constexpr int kQ2Part = 2;                               // tiles whose chains wait for one barrier
template <int DT>
constexpr int kRowPad = DT == DT_Q2_0 ? 2 : 4;  // columns between the blocks' terms (Q2_0: writes and reads both two words a bank)
// how a kernel's warps share a row: chains of Q2_0 (ONE) or not
template <int DT, bool ONE>
constexpr bool kChains = DT == DT_Q2_0 && ONE;
template <int DT, bool ONE>
constexpr int kRowWarps = kChains<DT, ONE> ? kQ2ChainWarps : RowFmt<DT>::kWarps;

__device__ __forceinline__ uint32_t rs32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool row_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Bounded; gives up at once where another warp already has.
__device__ __noinline__ bool row_wait_slow(uint32_t bar, uint32_t parity, volatile int *dead) {
    for (uint32_t i = 0; i < kRowSpin; i++) {
        if (row_try(bar, parity)) return true;
        if ((i & 1023u) == 0 && *dead) return false;
    }
    return false;
}
__device__ __noinline__ void row_drain(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 14) && !row_try(bar, parity); i++) {
    }
}
// d = A(16x32, u8) * B(32x8, s8) and d += A * B
__device__ __forceinline__ void mma_set(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_add(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_acc(bool set, int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (set)
        mma_set(d, a0, a1, a2, a3, b0, b1);
    else
        mma_add(d, a0, a1, a2, a3, b0, b1);
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// 16-bit x 8-bit pair products: a's halves (signed) with bytes 2, 3 (unsigned) of b; with bytes 0, 1 / 2, 3 (signed) of b
__device__ __forceinline__ int dp2a_hi_su(uint32_t a, uint32_t b) {
    int d;
    asm("dp2a.hi.s32.u32 %0, %1, %2, 0;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ int dp2a_ss(uint32_t a01, uint32_t a23, uint32_t b) {
    int d;
    asm("{\n\t.reg .s32 t;\n\tdp2a.lo.s32.s32 t, %1, %3, 0;\n\tdp2a.hi.s32.s32 %0, %2, %3, t;\n\t}" : "=r"(d) : "r"(a01), "r"(a23), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t pack16(int lo, int hi) { return __byte_perm((uint32_t)lo, (uint32_t)hi, 0x5410); }
__device__ __forceinline__ uint32_t lds16(const uint8_t *p) { return *reinterpret_cast<const unsigned short *>(p); }
__device__ __forceinline__ int sext8(uint32_t w, int k) { return (int)(int8_t)(w >> (8 * k)); }

// ---- what a lane (g = lane / 4, t = lane % 4) multiplies a unit by; kept in registers where a warp has one unit, else in the warp's
// own part of shared memory, a record of kActBytes per unit ----
template <int DT>
struct RowAct;
template <>
struct RowAct<DT_Q4K> {
    uint32_t c0, c1;  // codes 4t..4t+3 and 16+4t..+3 of sub-block g
    uint32_t bs;      // sums of the codes of sub-blocks 2t, 2t+1 (16 bits each)
    float d;
    __device__ __forceinline__ void put(uint8_t *p, int lane) const {
        reinterpret_cast<uint2 *>(p)[lane] = make_uint2(c0, c1);
        if (lane < 4) reinterpret_cast<uint2 *>(p + 256)[lane] = make_uint2(bs, __float_as_uint(d));
    }
    __device__ __forceinline__ void get(const uint8_t *p, int lane) {
        const uint2 c = reinterpret_cast<const uint2 *>(p)[lane], s = reinterpret_cast<const uint2 *>(p + 256)[lane & 3];
        c0 = c.x, c1 = c.y, bs = s.x, d = __uint_as_float(s.y);
    }
};
template <>
struct RowAct<DT_Q6K> {
    uint32_t c[2][2];   // [block][n]: codes 4t..4t+3 of sub-block 8n + g
    uint32_t bs[2][2];  // [block][n]: sums of sub-blocks 8n + 2t, 8n + 2t + 1
    float d[2];
    __device__ __forceinline__ void put(uint8_t *p, int lane) const {
        reinterpret_cast<uint4 *>(p)[lane] = make_uint4(c[0][0], c[0][1], c[1][0], c[1][1]);
        if (lane < 4) reinterpret_cast<uint4 *>(p + 512)[lane] = make_uint4(bs[0][0], bs[0][1], bs[1][0], bs[1][1]);
        if (lane == 0) *reinterpret_cast<float2 *>(p + 576) = make_float2(d[0], d[1]);
    }
    __device__ __forceinline__ void get(const uint8_t *p, int lane) {
        const uint4 v = reinterpret_cast<const uint4 *>(p)[lane], s = reinterpret_cast<const uint4 *>(p + 512)[lane & 3];
        const float2 e = *reinterpret_cast<const float2 *>(p + 576);
        c[0][0] = v.x, c[0][1] = v.y, c[1][0] = v.z, c[1][1] = v.w;
        bs[0][0] = s.x, bs[0][1] = s.y, bs[1][0] = s.z, bs[1][1] = s.w;
        d[0] = e.x, d[1] = e.y;
    }
};

// 8-bit codes of K elements of one block held by the warp (quantize_q8, crates/infr-cpu/src/quant.rs:27-58): a lane has 4 * NV of them
template <int NV>
__device__ __forceinline__ float quant_block(const float4 (&v)[NV], uint32_t (&codes)[NV]) {
    float am = 0.f;
#pragma unroll
    for (int i = 0; i < NV; i++) am = fmaxf(am, fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w))));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float d = am / 127.0f, id = d > 0.0f ? 1.0f / d : 0.0f;
#pragma unroll
    for (int i = 0; i < NV; i++) codes[i] = q8_codes4(v[i], id);
    return d;
}
// the sums that the quads 2t and 2t + 1 hold, packed
__device__ __forceinline__ uint32_t pair_sums(int s, int t) {
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return pack16(__shfl_sync(0xffffffffu, s, 8 * t), __shfl_sync(0xffffffffu, s, 8 * t + 4));
}

template <bool FUSED>
__device__ __forceinline__ void load_act(RowAct<DT_Q4K> &r, const Q8Dev &a, const float *x, int unit, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const size_t at = (size_t)unit * 256 + g * 32 + t * 4;
    if (FUSED) {
        const float4 v[2] = {*reinterpret_cast<const float4 *>(x + at), *reinterpret_cast<const float4 *>(x + at + 16)};
        uint32_t c[2];
        r.d = quant_block(v, c);
        r.c0 = c[0], r.c1 = c[1];
        r.bs = pair_sums(q8_sum4(c[0]) + q8_sum4(c[1]), t);
    } else {
        r.c0 = *reinterpret_cast<const uint32_t *>(a.qs + at);
        r.c1 = *reinterpret_cast<const uint32_t *>(a.qs + at + 16);
        const int2 s = *reinterpret_cast<const int2 *>(a.sums + (size_t)unit * 8 + 2 * t);
        r.bs = pack16(s.x, s.y);
        r.d = a.d[unit];
    }
}
template <bool FUSED>
__device__ __forceinline__ void load_act(RowAct<DT_Q6K> &r, const Q8Dev &a, const float *x, int unit, int lane) {
    const int g = lane >> 2, t = lane & 3;
    if (FUSED) {
        float4 v[2][2];
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int n = 0; n < 2; n++) v[b][n] = *reinterpret_cast<const float4 *>(x + (size_t)unit * 512 + b * 256 + n * 128 + g * 16 + t * 4);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            r.d[b] = quant_block(v[b], r.c[b]);
#pragma unroll
            for (int n = 0; n < 2; n++) r.bs[b][n] = pair_sums(q8_sum4(r.c[b][n]), t);
        }
    } else {
#pragma unroll
        for (int b = 0; b < 2; b++) {
#pragma unroll
            for (int n = 0; n < 2; n++) {
                r.c[b][n] = *reinterpret_cast<const uint32_t *>(a.qs + (size_t)unit * 512 + b * 256 + n * 128 + g * 16 + t * 4);
                const int2 s = *reinterpret_cast<const int2 *>(a.sums16 + (size_t)unit * 32 + b * 16 + n * 8 + 2 * t);
                r.bs[b][n] = pack16(s.x, s.y);
            }
            r.d[b] = a.d[unit * 2 + b];
        }
    }
}
// Q2_0: groups of 32 elements with a scale each, always in shared memory: group G's codes at 32 G as words [field f][word i] = elements
// 16i + f, 16i + 4 + f, 16i + 8 + f, 16i + 12 + f (the order in which a code word yields its fields), then per (half, t) the scales of
// groups 2t, 2t + 1 of the half and the negated sums of their codes.
__device__ __forceinline__ void load_q2(float4 (&v)[4], const float *x, int unit, int lane) {
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = *reinterpret_cast<const float4 *>(x + (size_t)unit * 512 + lane * 16 + k * 4);
}
template <bool FUSED>
__device__ __forceinline__ void put_act_q2(uint8_t *p, const Q8Dev &a, const float4 (&v)[4], int unit, int lane) {
    uint32_t w[4];
    float d;
    int sum;
    const int grp = lane >> 1, i = lane & 1;
    if (FUSED) {
        float am = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) am = fmaxf(am, fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w))));
        am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
        d = am / 127.0f;
        const float id = d > 0.0f ? 1.0f / d : 0.0f;
        sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            w[k] = q8_codes4(v[k], id);
            sum += q8_sum4(w[k]);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    } else {
        const uint4 v = *reinterpret_cast<const uint4 *>(a.qs + (size_t)unit * 512 + lane * 16);
        w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        d = a.d[(size_t)unit * 16 + grp];
        sum = a.sums[(size_t)unit * 16 + grp];
    }
    const uint32_t t01 = __byte_perm(w[0], w[1], 0x5140), t23 = __byte_perm(w[2], w[3], 0x5140);
    const uint32_t u01 = __byte_perm(w[0], w[1], 0x7362), u23 = __byte_perm(w[2], w[3], 0x7362);
    uint32_t *o = reinterpret_cast<uint32_t *>(p + grp * 32) + i;
    o[0] = __byte_perm(t01, t23, 0x5410);
    o[2] = __byte_perm(t01, t23, 0x7632);
    o[4] = __byte_perm(u01, u23, 0x5410);
    o[6] = __byte_perm(u01, u23, 0x7632);
    uint32_t *sc = reinterpret_cast<uint32_t *>(p + 512 + (grp >> 1) * 16);  // (half, t) = (grp / 8, grp % 8 / 2)
    if (i == 0)
        sc[grp & 1] = __float_as_uint(d);
    else
        sc[2 + (grp & 1)] = (uint32_t)-sum;
}

// A quad's four shares of rows g and g + 8 added up: lanes t = 0, 2 get row g, t = 1, 3 row g + 8.
__device__ __forceinline__ int quad_sum(const int (&v)[2], int t) {
    int s = ((t & 1) ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, (t & 1) ? v[0] : v[1], 1);
    return s + __shfl_xor_sync(0xffffffffu, s, 2);
}

// ---- one unit of 16 rows: the block's term in row g (t even) or g + 8 (t odd).  A block's integer sum is complete before it is converted
// and scaled, so every block contributes the CPU's value. ----
// Q4_K: columns 2p, 2p + 1 = sub-blocks of the low and the high nibbles of run p.  Of the bytes of a run only the low nibbles are masked out:
//   masked bytes x (codes of 2p in column 2p, NEGATED codes of 2p + 1 in column 2p + 1)  +  whole bytes x (codes of 2p + 1 in column 2p + 1)
// leaves 16 x the high nibbles' sum in column 2p + 1.  (The integer pipe has half rate: its instructions are what a unit costs, a mask per
// high nibble was 16 of 75.)
struct RowB4 {
    uint32_t lo[4][2], hi[4][2];
};
// bytes negated (each is within [-127, 127])
__device__ __forceinline__ uint32_t neg4(uint32_t v) { return __vneg4(v); }
__device__ __forceinline__ void select_q4k(const RowAct<DT_Q4K> &r, int g, RowB4 &b) {
    const uint32_t n0 = (g & 1) ? neg4(r.c0) : r.c0, n1 = (g & 1) ? neg4(r.c1) : r.c1, m0 = (g & 1) ? r.c0 : 0u, m1 = (g & 1) ? r.c1 : 0u;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const bool on = (g >> 1) == p;
        b.lo[p][0] = on ? n0 : 0u, b.lo[p][1] = on ? n1 : 0u, b.hi[p][0] = on ? m0 : 0u, b.hi[p][1] = on ? m1 : 0u;
    }
}
__device__ __forceinline__ float unit_q4k(const uint8_t *sl, int lane, const RowAct<DT_Q4K> &r, const RowB4 &b) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t at = rs32(sl) + ((lane & 7) + (lane & 8)) * 144 + 16 + (lane >> 4) * 16;
    int d0[4], d1[4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        uint32_t w[4];
        ldsm4(w, at + p * 32);
        mma_acc(p == 0, d1, w[0], w[1], w[2], w[3], b.hi[p][0], b.hi[p][1]);
        mma_acc(p == 0, d0, w[0] & 0x0F0F0F0Fu, w[1] & 0x0F0F0F0Fu, w[2] & 0x0F0F0F0Fu, w[3] & 0x0F0F0F0Fu, b.lo[p][0], b.lo[p][1]);
    }
    // get_scale_min_k4 (crates/infr-gguf/src/dequant.rs:73-83) of sub-blocks 2t, 2t + 1: scales in bytes 0, 1, mins in bytes 2, 3
    const uint32_t sel = (t & 1) ? 0x7632u : 0x5410u, m1 = t < 2 ? 0x3F3F3F3Fu : 0x30303030u, m2 = t < 2 ? 0u : 0x0F0F0F0Fu, sh = t < 2 ? 0u : 2u;
    const uint4 h[2] = {*reinterpret_cast<const uint4 *>(sl + g * 144), *reinterpret_cast<const uint4 *>(sl + (g + 8) * 144)};
    int sd[2], sm[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t k4 = ((__byte_perm(h[i].y, h[i].z, sel) >> sh) & m1) | (__byte_perm(h[i].w, h[i].w >> 4, sel) & m2);
        sd[i] = (int)__byte_perm(k4, 0, 0x4440) * d0[2 * i] + (int)__byte_perm(k4, 0, 0x4441) * ((d0[2 * i + 1] + d1[2 * i + 1]) >> 4);
        sm[i] = dp2a_hi_su(r.bs, k4);
    }
    const uint32_t dd = (t & 1) ? h[1].x : h[0].x;
    return __fmaf_rn(h2f(dd), (float)quad_sum(sd, t), -__fmul_rn(h2f(dd >> 16), (float)quad_sum(sm, t)));
}

// word at byte offset `off` (a multiple of 4) of a block that starts at p; ODD: p is 2 bytes past a word boundary
template <bool ODD>
__device__ __forceinline__ uint32_t word6(const uint8_t *p, int off) {
    if (!ODD) return *reinterpret_cast<const uint32_t *>(p + off);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(p + off - 2);
    return __funnelshift_r(q[0], q[1], 16);
}
// p0, p1: the block in rows g and g + 8
template <bool ODD>
__device__ __forceinline__ float2 block_q6k(const uint8_t *p0, const uint8_t *p1, int lane, const uint32_t (&code)[2], const uint32_t (&bs)[2], float d) {
    const int g = lane >> 2, t = lane & 3;
    int pr[2][4];  // [n]: column s = sub-block 8n + s
#pragma unroll
    for (int n = 0; n < 2; n++) {
        uint32_t a[4][4];  // [c][fragment word]: sub-blocks 8n + 2c (words 0, 1) and 8n + 2c + 1 (words 2, 3) of rows g, g + 8
#pragma unroll
        for (int j = 0; j < 2; j++) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint8_t *p = i ? p1 : p0;
                const int o = n * 64 + j * 16 + 4 * t;
                const uint32_t qa = word6<ODD>(p, o), qb = word6<ODD>(p, o + 32), qh = word6<ODD>(p, 128 + n * 32 + j * 16 + 4 * t);
                a[0][2 * j + i] = (qa & 0x0F0F0F0Fu) | ((qh << 4) & 0x30303030u);
                a[1][2 * j + i] = (qb & 0x0F0F0F0Fu) | ((qh << 2) & 0x30303030u);
                a[2][2 * j + i] = ((qa >> 4) & 0x0F0F0F0Fu) | (qh & 0x30303030u);
                a[3][2 * j + i] = ((qb >> 4) & 0x0F0F0F0Fu) | ((qh >> 2) & 0x30303030u);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; c++) mma_acc(c == 0, pr[n], a[c][0], a[c][1], a[c][2], a[c][3], g == 2 * c ? code[n] : 0u, g == 2 * c + 1 ? code[n] : 0u);
    }
    int isum[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint8_t *p = i ? p1 : p0;
        const uint32_t sc = lds16(p + 192 + 2 * t) | (lds16(p + 200 + 2 * t) << 16);  // int8 scales of sub-blocks 2t, 2t+1, 8+2t, 8+2t+1
        isum[i] = sext8(sc, 0) * pr[0][2 * i] + sext8(sc, 1) * pr[0][2 * i + 1] + sext8(sc, 2) * pr[1][2 * i] + sext8(sc, 3) * pr[1][2 * i + 1] -
                  32 * dp2a_ss(bs[0], bs[1], sc);
    }
    return make_float2(__fmul_rn(h2f(lds16(((t & 1) ? p1 : p0) + 208)), d), (float)quad_sum(isum, t));
}

// Half a Q2_0 unit (4 blocks of 64): lane t has block t of rows g, g + 8; the sums of its groups 2t, 2t + 1 end up in its own columns.
// dw: the block's scales in the two rows, s: 64 x the groups' sums.
// codes: this lane's groups for h = 0, 1 (zeros where another lane's column is meant), sc: scales and negated sums of groups 2t, 2t + 1.
__device__ __forceinline__ void half_q2(const uint8_t *p0, const uint8_t *p1, uint32_t mis, const uint4 *c0, const uint4 *c1, uint4 sc, float (&dw)[2], int (&s)[2][2]) {
    uint32_t c[2][4];
    const uint32_t sh = 16u + 8u * mis;  // 16, or 32 (= take the upper word)
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint32_t *q = reinterpret_cast<const uint32_t *>(i ? p1 : p0);
        const uint32_t w0 = q[0], w1 = q[1], w2 = q[2], w3 = q[3], w4 = q[4];
        dw[i] = h2f(w0 >> (8u * mis));
        c[i][0] = __funnelshift_rc(w0, w1, sh), c[i][1] = __funnelshift_rc(w1, w2, sh);
        c[i][2] = __funnelshift_rc(w2, w3, sh), c[i][3] = __funnelshift_rc(w3, w4, sh);
    }
    // field f of a code byte stays where it is: its products come out 4^f times too large; all are exact
    int d[4][4] = {{(int)sc.z, (int)sc.w, (int)sc.z, (int)sc.w}};
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint4 b01 = (h ? c1 : c0)[0], b23 = (h ? c1 : c0)[1];
        const uint32_t b[8] = {b01.x, b01.y, b01.z, b01.w, b23.x, b23.y, b23.z, b23.w};
#pragma unroll
        for (int f = 0; f < 4; f++) {
            const uint32_t m = 0x03030303u << (2 * f);
            mma_acc(f > 0 && h == 0, d[f], c[0][2 * h] & m, c[1][2 * h] & m, c[0][2 * h + 1] & m, c[1][2 * h + 1] & m, b[2 * f], b[2 * f + 1]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int k = 0; k < 2; k++) s[i][k] = ((d[0][2 * i + k] * 4 + d[1][2 * i + k]) * 4 + d[2][2 * i + k]) * 4 + d[3][2 * i + k];
}
// A block's two groups added to a chain: products of the scales, then one multiply-add each with the group's sum.
__device__ __forceinline__ float chain_q2(float chain, float dw, float sc0, float sc1, float sum0, float sum1) {
    return __fmaf_rn(__fmul_rn(dw, sc1), sum1, __fmaf_rn(__fmul_rn(dw, sc0), sum0, chain));
}

// Matrices with one in_f in one launch: their 16-row tiles follow each other in the CTAs' tile ranges.  NM > kSameRow: with a row each.
constexpr int kSameRow = 3;
template <int NM>
struct RowMats {
    CUtensorMap map[NM];
    float *y[NM];
    int out_f[NM];
    int tile_end[NM];                       // tiles of matrices 0..i
    int group[NM];                          // Q4_K, Q6_K: blocks added before their sum is added to the others'
    const float *x[NM > kSameRow ? NM : 1];
};
struct RowGeom {
    int units, upw;  // K units of a row, of a warp
    int slots;
    int tiles;
};

// ONE: a warp has one unit, its activations stay in registers; Q2_0: chains in registers (kChains).
template <int DT, int NM, bool FUSED, bool ONE, bool PUSH>
__global__ void __launch_bounds__(kRowWarps<DT, ONE> * 32, kChains<DT, ONE> ? 4 : 2)
    gemv_row_kernel(const __grid_constant__ RowMats<NM> mats, const Q8Dev a, const float *x, RowGeom geo, uint32_t *status,
                    const __grid_constant__ typename PushParam<PUSH>::type push) {
    using F = RowFmt<DT>;
    constexpr int kBox = kRowTile * F::kPitch;
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, kw = blockDim.x >> 5, S = geo.slots;
    uint8_t *acts = smem + (size_t)S * kw * kBox;                                                                       // [units][kActBytes]
    // sums that wait for a barrier, twice: chains [tile][warp][kQ2Chains], else terms [block][kPart * 16 + a pad], and the blocks' activation scales behind them
    constexpr int kPart = kChains<DT, ONE> ? kQ2Part : F::kPart, kCols = kPart * kRowTile, kStride = (kCols + kRowPad<DT>) * F::kTerm;
    constexpr int kBlocks = DT == DT_Q2_0 ? 8 : DT == DT_Q6K ? 2 : 1;
    float *parts = reinterpret_cast<float *>(acts + (ONE && DT != DT_Q2_0 ? 0 : (size_t)geo.units * F::kActBytes));
    const int buf = kChains<DT, ONE> ? kPart * kw * kQ2Chains : geo.units * kBlocks * kStride;  // of two buffers
    [[maybe_unused]] float *s_scale = parts + 2 * buf;
    __shared__ __align__(8) uint64_t s_bars[kRowWarps<DT, ONE> * kRowSlots];
    __shared__ __align__(16) uint32_t s_zero[8];
    __shared__ int s_dead;
    __shared__ uint32_t s_epoch;  // push mode: exchanges completed before this launch
    const uint8_t *ring = smem + (size_t)warp * S * kBox;
    const uint32_t bar0 = rs32(s_bars + warp * kRowSlots);
    if (lane == 0) {  // a warp's barriers are its own
        for (int i = 0; i < S; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x == 0) s_dead = 0;
    if (DT == DT_Q2_0 && threadIdx.x < 8) s_zero[threadIdx.x] = 0;
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int G = gridDim.x, base = geo.tiles / G, rem = geo.tiles % G;
    const int t_begin = blockIdx.x * base + (blockIdx.x < rem ? blockIdx.x : rem);
    const int n_tiles = base + (blockIdx.x < rem ? 1 : 0);
    // this warp's units: u0, u0 + kStep, ...
    constexpr int kStep = kChains<DT, ONE> ? 4 : 1;
    constexpr bool kOneUnit = ONE && DT != DT_Q2_0;
    const int u0 = kChains<DT, ONE> ? warp : warp * geo.upw;
    const int n_units = kOneUnit ? 1 : kChains<DT, ONE> ? (geo.units - warp + 3) / 4 : min(geo.upw, geo.units - u0);
    uint64_t policy;  // weights are read once a launch: they do not push what every CTA reads out of L2
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));

    // next box to fetch: unit i_unit of the 16 rows at i_row of matrix i_mat
    int i_left = n_tiles * n_units, i_unit = 0, i_mat = 0, i_row;
    {
        int T = t_begin;
        if (NM > 1) {
            while (T >= mats.tile_end[i_mat]) i_mat++;
            if (i_mat) T -= mats.tile_end[i_mat - 1];
        }
        i_row = T * kRowTile;
    }
    auto issue = [&](int slot) {
        if (i_left == 0) return;
        if (lane == 0) {
            const int unit = u0 + i_unit * kStep, col = DT == DT_Q6K ? ((unit * 420) & ~15) >> 1 : unit * 36;  // 16-bit / 32-bit elements of the map
            const uint32_t bar = bar0 + 8 * slot;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the slot come first
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kBox) : "memory");
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(
                             rs32(ring) + slot * kBox),
                         "l"(&mats.map[NM > 1 ? i_mat : 0]), "r"(col), "r"(i_row), "r"(bar), "l"(policy)
                         : "memory");
        }
        i_left--;
        if (kOneUnit || ++i_unit == n_units) {
            i_unit = 0;
            i_row += kRowTile;
            if (NM > 1 && i_mat < NM - 1 && i_row >= mats.out_f[i_mat]) i_row = 0, i_mat++;
        }
    };
    for (int s = 0; s < S; s++) issue(s);

    // ---- activations (from the launch before) ----
    [[maybe_unused]] const uint8_t *acts0 = acts;
    acts += (size_t)u0 * F::kActBytes;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (PUSH) {
        if (threadIdx.x == 0) s_epoch = *reinterpret_cast<const volatile uint32_t *>(push.ctrl);  // read after the barrier of a batch
    }
    int c_mat = 0, c_end = 0;  // the matrix whose row is in use, its last tile + 1
    if (NM > kSameRow) {
        while (t_begin >= mats.tile_end[c_mat]) c_mat++;
        c_end = mats.tile_end[c_mat];
        x = mats.x[c_mat];
    }
    [[maybe_unused]] RowAct<DT == DT_Q2_0 ? DT_Q4K : DT> act;
    [[maybe_unused]] RowB4 b4;
    auto take_row = [&]() {
        if constexpr (DT == DT_Q2_0) {
            auto put = [&](int u, const float4 (&v)[4]) { put_act_q2<FUSED>(acts + (size_t)u * kStep * F::kActBytes, a, v, u0 + u * kStep, lane); };
            float4 v0[4], v1[4];
            if (FUSED && ONE) {
                for (int u = 0; u < n_units; u += 2) {  // two units' loads in flight together
                    load_q2(v0, x, u0 + u * kStep, lane);
                    if (u + 1 < n_units) load_q2(v1, x, u0 + (u + 1) * kStep, lane);
                    put(u, v0);
                    if (u + 1 < n_units) put(u + 1, v1);
                }
            } else {
                for (int u = 0; u < n_units; u++) {
                    if (FUSED) load_q2(v0, x, u0 + u * kStep, lane);
                    put(u, v0);
                }
            }
            __syncwarp();
        } else if constexpr (ONE) {
            load_act<FUSED>(act, a, x, u0, lane);
        } else {
            int u = 0;
            for (; u + 2 <= n_units; u += 2) {  // two units' loads in flight together
                RowAct<DT> r0, r1;
                load_act<FUSED>(r0, a, x, u0 + u, lane);
                load_act<FUSED>(r1, a, x, u0 + u + 1, lane);
                r0.put(acts + (size_t)u * F::kActBytes, lane);
                r1.put(acts + (size_t)(u + 1) * F::kActBytes, lane);
            }
            if (u < n_units) {
                load_act<FUSED>(act, a, x, u0 + u, lane);
                act.put(acts + (size_t)u * F::kActBytes, lane);
            }
            __syncwarp();
        }
        if constexpr (DT == DT_Q4K && ONE) select_q4k(act, g, b4);
        if constexpr (DT == DT_Q4K) {
            if (ONE) {
                if (lane == 0) s_scale[u0] = act.d;
            } else {
                for (int u = lane; u < n_units; u += 32) s_scale[u0 + u] = reinterpret_cast<const float *>(acts + (size_t)u * F::kActBytes + 256)[1];
            }
        }
    };
    take_row();

    // ---- tiles ----
    int slot = 0;
    uint32_t ph = 0;
    int batch = 0;
    for (int b0 = 0, nb; b0 < n_tiles; b0 += nb) {
        float *sums = parts + (size_t)(batch & 1) * buf;
        nb = min(kPart, n_tiles - b0);
        if (NM > kSameRow) {  // a batch is of one row
            if (t_begin + b0 == c_end) {
                c_mat++;
                c_end = mats.tile_end[c_mat];
                x = mats.x[c_mat];
                __syncthreads();  // the scales of the last row are read
                take_row();
            }
            nb = min(nb, c_end - (t_begin + b0));
        }
        for (int k = 0; k < nb; k++) {
            [[maybe_unused]] float chain[2][2] = {{0.f, 0.f}, {0.f, 0.f}};                                    // Q2_0: [half][row g, g + 8]
            [[maybe_unused]] float *out0 = sums + u0 * kBlocks * kStride + (k * kRowTile + g + 8 * t) * F::kTerm;  // lanes t = 0, 1
            for (int u = 0; u < (kOneUnit ? 1 : n_units); u++) {
                if (!row_try(bar0 + 8 * slot, ph) && !row_wait_slow(bar0 + 8 * slot, ph, &s_dead)) {
                    // the launch's results are invalid: no more fetches, and those in flight land before the block gives its shared memory back
                    // (bounded; what is read from here on is in bounds)
                    s_dead = 1;
                    atomicExch(status, 3u);
                    i_left = 0;
                    for (int j = 0; j < S; j++) row_drain(bar0 + 8 * ((slot + j) % S), slot + j < S ? ph : ph ^ 1u);
                }
                const uint8_t *sl = ring + slot * kBox;
                if constexpr (DT == DT_Q4K) {
                    if (!ONE) {
                        act.get(acts + (size_t)u * F::kActBytes, lane);
                        select_q4k(act, g, b4);
                    }
                    const float x4 = unit_q4k(sl, lane, act, b4);
                    if (t < 2) out0[u * kStride] = x4;
                } else if constexpr (DT == DT_Q6K) {
                    if (!ONE) act.get(acts + (size_t)u * F::kActBytes, lane);
                    const uint8_t *p0 = sl + g * F::kPitch + 4 * ((u0 + u) & 3), *p1 = p0 + 8 * F::kPitch;
                    const float2 x0 = block_q6k<false>(p0, p1, lane, act.c[0], act.bs[0], act.d[0]);
                    const float2 x1 = block_q6k<true>(p0 + 210, p1 + 210, lane, act.c[1], act.bs[1], act.d[1]);
                    if (t < 2) {
                        *reinterpret_cast<float2 *>(out0 + 2 * u * kStride) = x0;
                        *reinterpret_cast<float2 *>(out0 + (2 * u + 1) * kStride) = x1;
                    }
                } else {
                    const uint8_t *rec = acts + (size_t)u * kStep * F::kActBytes;
                    const uint32_t mis = 2 * (t & 1);
                    const bool mine = t == (g >> 1);
                    const uint4 *zero = reinterpret_cast<const uint4 *>(s_zero);
#pragma unroll
                    for (int H = 0; H < 2; H++) {
                        float dw[2];
                        int s2[2][2];
                        const uint8_t *p0 = sl + g * 144 + H * 72 + 18 * t - mis;
                        const uint4 *cg = reinterpret_cast<const uint4 *>(rec + (8 * H + g) * 32);
                        const uint4 sc = *reinterpret_cast<const uint4 *>(rec + 512 + (4 * H + t) * 16);
                        half_q2(p0, p0 + 8 * 144, mis, mine && !(g & 1) ? cg : zero, mine && (g & 1) ? cg : zero, sc, dw, s2);
                        if (ONE) {
#pragma unroll
                            for (int i = 0; i < 2; i++)
                                chain[H][i] = chain_q2(chain[H][i], dw[i], __uint_as_float(sc.x), __uint_as_float(sc.y), (float)s2[i][0] * 0.015625f, (float)s2[i][1] * 0.015625f);
                        } else {  // (a sum has 14 bits)
                            float *o = sums + ((u0 + u) * 8 + 4 * H + t) * kStride + g * F::kTerm;
#pragma unroll
                            for (int i = 0; i < 2; i++)
                                *reinterpret_cast<float2 *>(o + i * 8 * F::kTerm) = make_float2(dw[i], __uint_as_float(pack16(s2[i][0] >> 6, s2[i][1] >> 6)));
                        }
                    }
                }
                __syncwarp();
                issue(slot);
                if (++slot == S) slot = 0, ph ^= 1u;
            }
            if constexpr (kChains<DT, ONE>) {
                float *p = sums + (k * kw + warp) * kQ2Chains + t * kQ2Stride + g;
                p[0] = chain[0][0], p[8] = chain[0][1];
                p[4 * kQ2Stride] = chain[1][0], p[4 * kQ2Stride + 8] = chain[1][1];
            }
        }
        __syncthreads();
        auto store = [&](int i, float v) {
            int T = t_begin + b0 + i / kRowTile, mi = 0;
            if (NM > 1) {
                while (T >= mats.tile_end[mi]) mi++;
                if (mi) T -= mats.tile_end[mi - 1];
            }
            const int row = T * kRowTile + i % kRowTile;
            if (row < mats.out_f[mi]) {
                if constexpr (PUSH)
                    push_store(push, s_epoch, (size_t)row, v);
                else
                    mats.y[mi][row] = v;
            }
        };
        auto add_term = [&](const float *col, int b, float acc) {
            if (DT == DT_Q4K) return __fmaf_rn(s_scale[b], col[b * kStride], acc);
            const float2 x2 = *reinterpret_cast<const float2 *>(col + b * kStride);
            return __fmaf_rn(x2.x, x2.y, acc);
        };
        const int blocks = geo.units * kBlocks;
        if constexpr (DT == DT_Q2_0 && !ONE) {
            // a warp a result, a lane a chain
            for (int i = warp; i < kRowTile; i += kw) {
                float v = 0.f;
#pragma unroll 4
                for (int b = lane; b < blocks; b += 32) {
                    const float2 x2 = *reinterpret_cast<const float2 *>(sums + b * kStride + i * F::kTerm);
                    const float2 sc = *reinterpret_cast<const float2 *>(acts0 + (b >> 3) * F::kActBytes + 512 + (b & 7) * 16);
                    const uint32_t s2 = __float_as_uint(x2.y);
                    v = chain_q2(v, x2.x, sc.x, sc.y, (float)(int)(short)(s2 & 0xFFFFu), (float)((int)s2 >> 16));
                }
                v = warp_sum(v);
                if (lane == 0) store(i, v);
            }
        } else if constexpr (DT == DT_Q2_0) {
            // eight threads a result: chains j, j + 8, j + 16, j + 24 (one of each class), then across the threads
            for (int i = threadIdx.x >> 3; i < nb * kRowTile; i += blockDim.x >> 3) {
                const float *p = sums + i / kRowTile * kw * kQ2Chains + (threadIdx.x & 7) * kQ2Stride + i % kRowTile;
                float v[4];
#pragma unroll
                for (int c = 0; c < 4; c++) v[c] = c < kw ? p[c * kQ2Chains] : 0.f;
                float s = (v[0] + v[2]) + (v[1] + v[3]);
#pragma unroll
                for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if ((threadIdx.x & 7) == 0) store(i, s);
            }
        } else if constexpr (!ONE) {
            // Long rows: eight threads a result, each adds groups of blocks in order, and the groups are added in order (14336 -> 4096: 8.0 us,
            // with one thread a result 8.8).  A warp's four results are of one tile.
            for (int i = threadIdx.x >> 3; i < nb * kRowTile; i += blockDim.x >> 3) {
                int mi = 0;
                if (NM > 1)
                    while (t_begin + b0 + i / kRowTile >= mats.tile_end[mi]) mi++;
                const int gs = mats.group[mi], q = threadIdx.x & 7;
                const float *col = sums + i * F::kTerm;
                float part[2] = {0.f, 0.f}, v = 0.f;  // groups q and q + 8: at most 16
#pragma unroll
                for (int h = 0; h < 2; h++)
                    for (int b = (q + 8 * h) * gs; b < min(blocks, (q + 8 * h + 1) * gs); b++) part[h] = add_term(col, b, part[h]);
#pragma unroll
                for (int h = 0; h < 2; h++)
                    if (h == 0 || blocks > 8 * gs)
#pragma unroll
                        for (int gr = 0; gr < 8; gr++) v += __shfl_sync(0xffffffffu, part[h], gr, 8);
                if (q == 0) store(i, v);
            }
        } else {
            // A thread a result, on two warps (Q6_K: one) that change from batch to batch; the others go on (two buffers of sums).
            for (int i = (int)threadIdx.x - batch * kCols % (int)blockDim.x; i < nb * kRowTile; i += blockDim.x) {
                if (i < 0) i += blockDim.x;
                if (i >= nb * kRowTile) break;
                const float *col = sums + i * F::kTerm;
                int mi = 0;
                if (NM > 1)
                    while (t_begin + b0 + i / kRowTile >= mats.tile_end[mi]) mi++;
                const int gs = mats.group[mi];
                float v = 0.f, acc = 0.f;
                int left = gs;
#pragma unroll 4
                for (int b = 0; b < blocks; b++) {
                    acc = add_term(col, b, acc);
                    if (--left == 0 || b == blocks - 1) v += acc, acc = 0.f, left = gs;
                }
                store(i, v);
            }
        }
        batch++;
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn row_encode() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

template <int DT>
bool row_map(CUtensorMap *map, const uint8_t *w, int units, int rows) {
    EncodeTiledFn enc = row_encode();
    if (!enc) return false;
    constexpr bool q6 = DT == DT_Q6K;
    const cuuint64_t bytes = (cuuint64_t)units * (q6 ? 420 : 144);
    const cuuint64_t gdim[2] = {bytes / (q6 ? 2 : 4), (cuuint64_t)rows}, gstride[1] = {bytes};
    const cuuint32_t box[2] = {(cuuint32_t)RowFmt<DT>::kPitch / (q6 ? 2 : 4), (cuuint32_t)kRowTile}, estr[2] = {1, 1};
    return enc(map, q6 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t *>(w), gdim, gstride, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Lets a kernel have all the shared memory there is, once per device (0.5 us of a call's 4.5 when set on each launch).  Setting it again
// from another thread meanwhile changes nothing.
template <int DT, int NM, bool FUSED, bool ONE, bool PUSH>
std::atomic<uint64_t> allowed{0};
cudaError_t allow_smem(const void *kernel, const DeviceInfo &dev, std::atomic<uint64_t> &done) {
    int id = 0;
    cudaError_t e = cudaGetDevice(&id);
    if (e != cudaSuccess || (id < 64 && (done.load(std::memory_order_acquire) >> id) & 1)) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kernel);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.max_smem_optin - (int)fa.sharedSizeBytes);
    // all of the SM's memory as shared memory, so that the launches around this one find room beside it
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess && id < 64) done.fetch_or(1ull << id, std::memory_order_release);
    return e;
}

template <int DT, int NM, bool FUSED, bool ONE, bool PUSH>
cudaError_t launch_row(const RowMats<NM> &mats, const Q8Dev &a, const float *x, RowGeom geo, int kw, const DeviceInfo &dev, uint32_t *status, cudaStream_t st,
                       const typename PushParam<PUSH>::type &push) {
    using F = RowFmt<DT>;
    const size_t cols = F::kPart * kRowTile, blocks = (size_t)geo.units * (DT == DT_Q2_0 ? 8 : DT == DT_Q6K ? 2 : 1);
    const size_t fixed = (ONE && DT != DT_Q2_0 ? 0 : (size_t)geo.units * F::kActBytes) +
                         (kChains<DT, ONE> ? 2 * (size_t)kQ2Part * kw * kQ2Chains : 2 * blocks * (cols + kRowPad<DT>) * F::kTerm + (DT == DT_Q4K ? blocks : 0)) * 4;
    const size_t per_slot = (size_t)kw * kRowTile * F::kPitch;
    // Several CTAs a SM where rows are short and each has a tile: more warps at work, but each CTA reads (or quantises) the row for itself.
    // (us with one CTA a SM / as many as have a tile: Q4_K 2048 -> 5632 3.0 / 2.5.  Chains of Q2_0 also where only some SMs have two tiles, four
    // warps are few: codes 4096 -> 4096 3.7 / 3.1, 14336 -> 4096 9.4 / 7.0, 3072 -> 8192 4.3 / 3.6.)
    int per_sm = F::kWarps / kw;
    int want = geo.tiles / dev.sm_count;
    if (kChains<DT, ONE> && geo.tiles % dev.sm_count) want++;
    if (per_sm > want) per_sm = want < 1 ? 1 : want;
    while (per_sm > 1 && (fixed + 2 * per_slot + 1024) * per_sm > (size_t)dev.max_smem_optin + 1024) per_sm--;
    const int grid = geo.tiles < dev.sm_count * per_sm ? geo.tiles : dev.sm_count * per_sm;
    // Two slots, no more than a warp has units; three for long Q4_K rows, whose warps fetch neighbouring units (14336 -> 4096 8.8 / 8.1 us;
    // 4096 -> 128256, where they fetch tiles far apart, 50 / 56).
    int slots = (geo.tiles + grid - 1) / grid * geo.upw;
    if (slots > (DT == DT_Q4K && geo.upw > 1 ? 3 : 2)) slots = DT == DT_Q4K && geo.upw > 1 ? 3 : 2;
    if (fixed + slots * per_slot > (size_t)dev.max_smem_optin - 2048) slots = 1;
    size_t smem = fixed + slots * per_slot;
    // No more than per_sm CTAs fit on a SM, so that the CTAs of a launch spread evenly whatever the launch before still holds.  (With room for
    // two where one is meant, some SMs got two and others none: gate and up of a decoded token 40 us instead of 13, in a chain with other
    // kernels; a chain of this kernel alone is as fast either way.)
    const size_t least = ((size_t)dev.max_smem_optin + 1024) / (per_sm + 1) - 1024;
    if (smem < least) smem = least;
    if (smem > (size_t)dev.max_smem_optin - 2048) return cudaErrorInvalidValue;
    geo.slots = slots;
    auto kernel = gemv_row_kernel<DT, NM, FUSED, ONE, PUSH>;
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(kernel), dev, allowed<DT, NM, FUSED, ONE, PUSH>);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)kw * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, mats, a, x, geo, status, push);
}

// Blocks of a row that are added before their sum is added to the others': the K split over 4, 8 or 16 warps that the kernels for two rows and
// more (gemv_mma.cu, gemv_mma_q6.cu) choose by the number of 16-row tiles and by what fits beside `nb` blocks of one staged row, so that a
// result keeps the bits it has there.
int row_group(int dt, int nb, int tiles, const DeviceInfo &dev) {
    const size_t top = (size_t)dev.max_smem_optin;
    auto need = [&](int kw, int units) {  // shared memory with `units` ring slots of a block a warp
        return (size_t)nb * (dt == DT_Q4K ? 368 : 384) + (size_t)kw * 1056 + 64 + (size_t)units * kw * kRowTile * (dt == DT_Q4K ? 144 : 224);
    };
    auto two = [&](int kw) { return need(kw, dt == DT_Q4K && (nb + kw - 1) / kw > 1 ? 4 : 2); };
    const int kw0 = tiles > 2 * dev.sm_count ? 4 : tiles > dev.sm_count ? 8 : 16;
    int kw = kw0;
    if (dt == DT_Q6K && kw == 4 && need(4, 3) > top / 4 - 2048) kw = 8;
    while (kw < 16 && two(kw) > top / (16 / kw) - 2048) kw *= 2;
    while (kw > 4 && kw > nb) kw /= 2;
    while (kw > 4 && two(kw) > top - 1024) kw /= 2;
    if (dt == DT_Q4K && kw == 16 && kw0 < 16 && nb >= 8 && need(8, 2) <= top / 2 - 2048) kw = 8;
    return (nb + kw - 1) / kw;
}

template <int DT, int NM>
cudaError_t launch_row_dt(const GemvRow &d, const DeviceInfo &dev, uint32_t *status, cudaStream_t st, const GemvPush *push) {
    using F = RowFmt<DT>;
    RowGeom geo{d.in_f / F::kUnit, 0, 0, 0};
    RowMats<NM> mats;
    memset(&mats, 0, sizeof mats);
    for (int i = 0; i < d.n; i++) {
        if (!row_map<DT>(&mats.map[i], d.mats[i].w, geo.units, d.mats[i].out_f)) return cudaErrorInvalidValue;
        mats.y[i] = d.mats[i].y;
        mats.out_f[i] = d.mats[i].out_f;
        geo.tiles += (d.mats[i].out_f + kRowTile - 1) / kRowTile;
        mats.tile_end[i] = geo.tiles;
        if constexpr (NM > kSameRow) mats.x[i] = d.mats[i].x;
    }
    for (int i = d.n; i < NM; i++) mats.tile_end[i] = geo.tiles;
    auto split = [&](int warps) {
        geo.upw = (geo.units + warps - 1) / warps;
        return (geo.units + geo.upw - 1) / geo.upw;
    };
    if constexpr (DT != DT_Q2_0) {
        auto tiles = [](int rows) { return (rows + kRowTile - 1) / kRowTile; };
        for (int i = 0; i < d.n; i++)
            mats.group[i] = row_group(DT, d.in_f / 256, DT == DT_Q4K ? tiles(d.mats[i].out_f) + tiles(d.mats[i].with) : tiles(d.mats[i].out_f), dev);
    }
    const Q8Dev none{nullptr, nullptr, nullptr, nullptr, 0};
    const int kw = split(F::kWarps);
    bool one = geo.upw == 1;
    if constexpr (DT == DT_Q2_0) {
        // Chains in four warps a CTA; long rows whose CTAs have a tile or so each: more warps a row, the blocks' sums in shared memory (us a call,
        // chains / sums: codes 14336 -> 1024 5.7 / 4.4, -> 4096 7.0 / 8.2, f32 rows 14336 -> 1024 9.0 / 5.8, -> 4096 10.6 / 9.5, -> 8192 14.6 / 15.5;
        // 4096 -> 1024 3.2 / 3.0, -> 4096 4.1 / 4.8).
        one = geo.units <= 8 || geo.tiles > (d.codes ? 1 : 2) * dev.sm_count;
    }
#define INFR_ROW(FUSED_, PUSH_, A_, P_)                                                                                              \
    do {                                                                                                                             \
        if (!one) {                                                                                                                  \
            const cudaError_t e = launch_row<DT, NM, FUSED_, false, PUSH_>(mats, A_, d.x, geo, kw, dev, status, st, P_);             \
            if (DT != DT_Q2_0 || e != cudaErrorInvalidValue || geo.tiles <= dev.sm_count) return e;                                  \
            cudaGetLastError(); /* the row's blocks leave no room */                                                                 \
        }                                                                                                                            \
        const int w = DT == DT_Q2_0 ? (geo.units < kQ2ChainWarps ? geo.units : kQ2ChainWarps) : kw;                                   \
        if (DT == DT_Q2_0) geo.upw = (geo.units + w - 1) / w;                                                                        \
        return launch_row<DT, NM, FUSED_, true, PUSH_>(mats, A_, d.x, geo, w, dev, status, st, P_);                                  \
    } while (0)
    if constexpr (NM > kSameRow) {
        INFR_ROW(true, false, none, NoPush{});
    } else {
        if (push) {
            if constexpr (NM == 1 && DT != DT_Q2_0) INFR_ROW(false, true, *d.codes, *push);
            return cudaErrorInvalidValue;
        }
        if (d.codes) INFR_ROW(false, false, *d.codes, NoPush{});
        INFR_ROW(true, false, none, NoPush{});
    }
#undef INFR_ROW
}

}  // namespace

bool gemv_row_takes(int dt, int in_f) {
    if (in_f < 1) return false;
    return dt == DT_Q4K ? in_f % 256 == 0 : dt == DT_Q6K ? in_f % 2048 == 0 : dt == DT_Q2_0 && in_f % 512 == 0;
}

cudaError_t launch_gemv_row(const GemvRow &d, const DeviceInfo &dev, uint32_t *status, cudaStream_t st, const GemvPush *push) {
    const int dt = d.dtype;
    if (!gemv_row_takes(dt, d.in_f) || d.n < 1 || d.n > kGemvRowMats || (push && (!d.codes || d.n != 1))) return cudaErrorInvalidValue;
    const bool own_rows = !d.codes && !d.x;
    if (!own_rows && d.n > kSameRow) return cudaErrorInvalidValue;
    if (d.codes && (d.codes->gran != act_gran(dt) || (dt == DT_Q6K && !d.codes->sums16))) return cudaErrorInvalidValue;
    if (d.x && (uintptr_t)d.x % 16) return cudaErrorInvalidValue;
    for (int i = 0; i < d.n; i++)
        if (d.mats[i].out_f < 1 || (own_rows && (!d.mats[i].x || (uintptr_t)d.mats[i].x % 16))) return cudaErrorInvalidValue;
#define INFR_ROW_DT(N)                                                                         \
    do {                                                                                       \
        if (dt == DT_Q4K) return launch_row_dt<DT_Q4K, N>(d, dev, status, st, push);           \
        if (dt == DT_Q6K) return launch_row_dt<DT_Q6K, N>(d, dev, status, st, push);           \
        return launch_row_dt<DT_Q2_0, N>(d, dev, status, st, push);                            \
    } while (0)
    if (own_rows) INFR_ROW_DT(kGemvRowMats);
    if (d.n == 1) INFR_ROW_DT(1);
    if (d.n == 2) INFR_ROW_DT(2);
    INFR_ROW_DT(3);
#undef INFR_ROW_DT
}

}  // namespace infr
