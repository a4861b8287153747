// The ops of a dense decode step that sit between the quantized Linears: RMSNorm (optionally fused with the
// residual add in front of it), RoPE, the f16 KV-cache write (optionally fused with RoPE of q and k), causal
// attention over an f16 KV cache with the keys split over CTAs, the SiLU gate, the residual add and argmax.
// Semantics follow the reference's CPU backend op by op (crates/infr-cpu/src/lib.rs: RmsNorm 801-825, Rope
// 1493-1553, WriteKv 1635-1673, Attention 1744-1888, GatedAct 1890-1944, Add 1972-1987, Argmax 2167-2187).
// All of them are HBM- or latency-bound elementwise / reduction kernels; every kernel waits for its producer
// with `griddepcontrol.wait` before its first read, so a chain of them can overlap launch with the tail of
// the previous kernel.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kernels.h"

#include "pdl.cuh"
#include "q8_code.cuh"
#include "row_norm.cuh"

namespace infr {
namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ---------------------------------------------------------------------------------------------- RMSNorm
// One CTA per row.  With ADD the row is a + b, which is also written to sum_dst (the residual stream).
template <bool ADD>
__global__ void __launch_bounds__(1024) rms_norm_kernel(const float *a, const float *b, float *sum_dst,  // sum_dst may alias a
                                                        const float *__restrict__ w, float *__restrict__ dst, int dim, float eps) {
    __shared__ float s_part[32];
    __shared__ float s_scale;
    pdl_go();
    pdl_wait();
    const size_t base = (size_t)blockIdx.x * dim;
    const int n4 = (dim & 3) ? 0 : dim >> 2;  // 16-byte accesses only when every row starts on a 16-byte boundary
    float ss = 0.f;
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        float4 v = reinterpret_cast<const float4 *>(a + base)[i];
        if (ADD) {
            const float4 u = reinterpret_cast<const float4 *>(b + base)[i];
            v.x += u.x, v.y += u.y, v.z += u.z, v.w += u.w;
            reinterpret_cast<float4 *>(sum_dst + base)[i] = v;
        }
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    for (int i = (n4 << 2) + threadIdx.x; i < dim; i += blockDim.x) {
        float v = a[base + i];
        if (ADD) {
            v += b[base + i];
            sum_dst[base + i] = v;
        }
        ss += v * v;
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x < 32) {
        float t = threadIdx.x < (blockDim.x + 31) / 32 ? s_part[threadIdx.x] : 0.f;
        t = warp_sum(t);
        if (threadIdx.x == 0) s_scale = 1.0f / sqrtf(t / (float)dim + eps);
    }
    __syncthreads();
    const float s = s_scale;
    const float *src = ADD ? sum_dst : a;  // a thread re-reads only what it wrote itself
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(src + base)[i];
        const float4 g = reinterpret_cast<const float4 *>(w)[i];
        reinterpret_cast<float4 *>(dst + base)[i] = make_float4(v.x * s * g.x, v.y * s * g.y, v.z * s * g.z, v.w * s * g.w);
    }
    for (int i = (n4 << 2) + threadIdx.x; i < dim; i += blockDim.x) dst[base + i] = src[base + i] * s * w[i];
}

// ---------------------------------------------------------------------------------------------- RoPE
// theta^(-2p/rope_dim): the exponent is formed in f32 like the reference's, the power in f64 and rounded once,
// which is what a correctly rounded f32 powf returns.
__device__ __forceinline__ float rope_freq(float theta, int p, int rope_dim) {
    const float e = -2.0f * (float)p / (float)rope_dim;
    return (float)pow((double)theta, (double)e);
}

__device__ __forceinline__ void rope_pair(float a, float b, float ang, float *oa, float *ob) {
    const float sn = sinf(ang), c = cosf(ang);
    *oa = a * c - b * sn;
    *ob = a * sn + b * c;
}

// thread = (row, head, pair or pass-through element)
__global__ void __launch_bounds__(256) rope_kernel(const float *x, const int32_t *positions,
                                                   float *__restrict__ dst, int rows, int n_head, int head_dim, int rope_dim,
                                                   float theta, int neox) {
    pdl_go();
    pdl_wait();
    const int hf = rope_dim / 2, per_head = hf + (head_dim - rope_dim);
    const size_t total = (size_t)rows * n_head * per_head;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int e = (int)(i % per_head);
        const size_t rh = i / per_head;
        const int r = (int)(rh / n_head);
        const size_t b = rh * head_dim;
        if (e < hf) {
            const int i0 = neox ? e : 2 * e, i1 = neox ? e + hf : 2 * e + 1;
            const float ang = (float)positions[r] * rope_freq(theta, e, rope_dim);
            float oa, ob;
            rope_pair(x[b + i0], x[b + i1], ang, &oa, &ob);
            dst[b + i0] = oa;
            dst[b + i1] = ob;
        } else {
            const int j = rope_dim + (e - hf);
            dst[b + j] = x[b + j];
        }
    }
}

// RoPE of q in place, RoPE of k straight into the f16 K cache, v into the f16 V cache: one launch instead of
// Rope, Rope, WriteKv, WriteKv (crates/infr-llama/src/seam/runner.rs:3611-3656).  Row r belongs to sequence
// r / rows_per_seq, whose caches start seq_stride elements after the previous sequence's, and lands at cache
// row positions[r].  Full-head rotation only (rope_dim == head_dim).
constexpr int kRopeTable = 128;  // frequencies a block keeps
constexpr int kPageRows = 128;  // rows of a page of a paged KV cache = keys of an attention tile
__global__ void __launch_bounds__(256) rope_write_kv_kernel(float *__restrict__ q, const float *k, const float *v,
                                                            const int32_t *positions, __half *__restrict__ k_cache,
                                                            __half *__restrict__ v_cache, int rows, int n_head, int n_kv, int head_dim,
                                                            float theta, int neox, int rows_per_seq, size_t seq_stride, int write_pos,
                                                            const int32_t *block_table, int table_stride, int n_pages) {
    // The frequencies (f64 powers) depend on nothing before: a block forms each once, before the wait.  (Longer heads: one by one.)
    __shared__ float s_freq[kRopeTable];
    pdl_go();
    const int hf = head_dim / 2;
    const bool table = hf <= kRopeTable;
    if (table)
        for (int p = threadIdx.x; p < hf; p += blockDim.x) s_freq[p] = rope_freq(theta, p, head_dim);
    __syncthreads();
    auto freq = [&](int p) { return table ? s_freq[p] : rope_freq(theta, p, head_dim); };
    pdl_wait();
    const size_t nq = (size_t)rows * n_head * hf, nk = (size_t)rows * n_kv * hf, total = nq + 2 * nk;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        if (i < nq) {
            const int p = (int)(i % hf);
            const size_t rh = i / hf;
            const int r = (int)(rh / n_head);
            const size_t b = rh * head_dim;
            const int i0 = neox ? p : 2 * p, i1 = neox ? p + hf : 2 * p + 1;
            float oa, ob;
            rope_pair(q[b + i0], q[b + i1], (float)positions[r] * freq(p), &oa, &ob);
            q[b + i0] = oa;
            q[b + i1] = ob;
        } else {
            const bool is_v = i >= nq + nk;
            const size_t t = i - nq - (is_v ? nk : 0);
            const int p = (int)(t % hf);
            const size_t rh = t / hf;  // row * n_kv + head
            const int r = (int)(rh / n_kv), h = (int)(rh % n_kv);
            const size_t b = rh * head_dim;
            // cache row: the op's own `pos` + row when the caller gives one (Op::WriteKv), else the row's position
            const size_t crow = write_pos >= 0 ? (size_t)(write_pos + r % rows_per_seq) : (size_t)positions[r];
            size_t cb;
            if (block_table) {  // paged caches: row crow of the sequence lives in page table[seq][crow / 128] of the pool
                const int pg = min(max(block_table[(size_t)(r / rows_per_seq) * table_stride + crow / kPageRows], 0), n_pages - 1);
                cb = (((size_t)pg * kPageRows + crow % kPageRows) * n_kv + h) * head_dim;
            } else {
                cb = (size_t)(r / rows_per_seq) * seq_stride + (crow * n_kv + h) * head_dim;
            }
            if (is_v) {
                v_cache[cb + 2 * p] = __float2half_rn(v[b + 2 * p]);
                v_cache[cb + 2 * p + 1] = __float2half_rn(v[b + 2 * p + 1]);
            } else {
                const int i0 = neox ? p : 2 * p, i1 = neox ? p + hf : 2 * p + 1;
                float oa, ob;
                rope_pair(k[b + i0], k[b + i1], (float)positions[r] * freq(p), &oa, &ob);
                k_cache[cb + i0] = __float2half_rn(oa);
                k_cache[cb + i1] = __float2half_rn(ob);
            }
        }
    }
}

__global__ void __launch_bounds__(256) write_kv_kernel(const float *src, __half *__restrict__ cache, size_t n) {
    pdl_go();
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        cache[i] = __float2half_rn(src[i]);
}

// ---------------------------------------------------------------------------------------------- attention
constexpr int kAttnTile = 128;     // keys per CTA
constexpr int kAttnThreads = 256;  // eight warps: 16 keys each in the score phase, 16 output dims each in the value phase

// CTA = (key tile, KV head, query row).  The tile's 128 key rows and 128 value rows (head_dim halves each) are
// copied into shared memory, all copies of the CTA in flight together and none in a register.
//
// Both products run on the warp-level matrix unit in f16 WITHOUT giving up f32 operands: the cache values are f16, and the f32 operand (q,
// then the softmax weights p) is split into two f16 pieces, hi = its top 11 significant bits, mid = the next 11 of the remainder times 2^11,
// which sit in two neighbouring columns of the instruction's N dimension and are added afterwards; what is dropped is below 2^-22 of the
// operand, the size of the rounding of an f32 accumulation itself.  A power of two per head brings the largest |q| to 2^14 .. 2^15, weights
// (at most 1) are multiplied by 2^15: an element down to 2^-26 of the largest keeps all these bits.  A tile with an element below that (f16 ends
// there) is multiplied in tf32 pieces, which have the exponents of f32 (tile_tf32): every element keeps its bits, whatever the others are.
// Products are exact, sums are f32.  (The same split in tf32 pieces, with the same bits, has to widen every half of the tile to 32 bits first: a batch of 32 sequences at 4097 keys 113 -> 95 us a layer.)
// Phase 1: warp w scores keys 16w..16w+15 against the G query heads that share the KV head: A = the keys (ldmatrix),
// B = the q pieces, K = head_dim in steps of 8.  Phase 2: one warp per head turns the tile's scores into
// exp(s - m), their sum, and the two pieces of each weight.  Phase 3: warp w owns output dims 16 (w mod HD/16):
// A = the values transposed (ldmatrix.trans), B = the weight pieces, K = the keys in steps of 8; with head_dim 64 the
// two halves of the keys go to two warps and meet in shared memory (over the key tile, dead by then).  The tile's
// (m, l, o) goes to the workspace for the merge kernel.
// A tile's keys or values in shared memory: kAttnTile rows of HD halves.  frag: the 16-byte piece 2 j + hi (hi = 0, 1) of a row;
// that of the row 8 n rows on is 8 n kStride bytes on.  Either way the eight rows
// of an ldmatrix lie in distinct banks.
template <int HD>
struct PaddedTile {  // rows 16 bytes past a multiple of 128
    static constexpr int kStride = HD * 2 + 16, kBytes = kAttnTile * kStride, kAlign = 16;
    static __device__ __forceinline__ uint8_t *frag(uint8_t *tile, int row, int hi, int j) { return tile + row * kStride + hi * 16 + j * 32; }
};
template <int HD>
struct BoxedTile {  // as tensor copies of rows x 64 halves with the 128-byte swizzle leave it, the first 64 dims first
    static constexpr int kStride = 128, kBytes = kAttnTile * HD * 2, kAlign = 1024;
    static __device__ __forceinline__ uint8_t *frag(uint8_t *tile, int row, int hi, int j) {
        return tile + row * 128 + (j >> 2) * (kAttnTile * 128) + ((((hi ^ row) & 7) << 4) ^ ((j & 3) << 5));
    }
};
constexpr int kBoxRows = 16;
__device__ __forceinline__ int boxed_rows(int keys) { return (keys + kBoxRows - 1) / kBoxRows * kBoxRows; }
// dynamic shared memory from a multiple of the tile's alignment on
template <class T>
__device__ __forceinline__ uint8_t *align_tile(uint8_t *p) {
    if constexpr (T::kAlign <= 16) return p;
    return p + (-(uint32_t)__cvta_generic_to_shared(p) & (T::kAlign - 1));
}
template <class T>
constexpr int kTileBytes = 2 * T::kBytes + T::kAlign - 16;
// Maps of the caches (rows of n_kv * HD halves): keys and values in boxes of a whole tile's rows, the same in boxes of kBoxRows.
struct AttnMaps {
    CUtensorMap map[4];
};
struct NoMaps {};
// By one thread; by the whole CTA with the maps
template <int HD>
__device__ __forceinline__ void init_bars(uint64_t *s_bar) {
#pragma unroll
    for (int i = 0; i < 2; i++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(s_bar + i)), "n"(HD / 64) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
template <int HD>
__device__ __forceinline__ void init_bars(uint64_t *s_bar, const AttnMaps &maps) {
    if (threadIdx.x % 32 == 0 && threadIdx.x < 128) asm volatile("prefetch.tensormap [%0];" ::"l"(maps.map + threadIdx.x / 32) : "memory");
    if (threadIdx.x == 0) init_bars<HD>(s_bar);
}
// Warps 0 .. HD / 32 - 1 fetch a tile, from row `row0` of a sequence's caches on: warp w the dims 64 (w / 2) .. + 63 of the keys (even) or values, in one copy; of a tile of
// fewer than 128 keys the boxes with keys.  What bounds a batch's attention is how many bytes an SM has on their way, three tiles at most: the time a tile takes to
// ask for its bytes counts in full.  32 sequences at 4097 keys, us a call with the merge: a bulk copy for every row (a warp issues those of its lanes one
// after the other) 102.6; 16 boxes a warp 98; this 91.8 (skeleton without arithmetic: 89).  head_dim 64, 16 heads / 16: 130 -> 90.
template <int HD>
__device__ __forceinline__ void fetch_tile(const AttnMaps &maps, uint8_t *s_k, uint8_t *s_v, uint64_t *s_bar, int kvh, int row0, int seq, int keys) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, which = warp & 1, half = warp >> 1;
    if (half >= HD / 64) return;
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(s_bar + which), to = (uint32_t)__cvta_generic_to_shared(which ? s_v : s_k) + half * (kAttnTile * 128);
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"((uint32_t)(boxed_rows(keys) * 128)) : "memory");
    __syncwarp();
    auto copy = [&](const CUtensorMap *map, int first) {
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(to + first * 128), "l"(map),
                     "r"(kvh * HD + half * 64), "r"(row0 + first), "r"(seq), "r"(b)
                     : "memory");
    };
    if (keys == kAttnTile) {
        if (lane == 0) copy(maps.map + which, 0);
    } else if (lane * kBoxRows < keys) {
        copy(maps.map + 2 + which, lane * kBoxRows);
    }
}
// Rows r0 .. r1 - 1 of the values, past the end of a tile: the matrix unit is to multiply 0 (not stale bits) by the weight 0.  Those of a box that
// is fetched once it has landed, the others at once.  (Scores past the end are not looked at.)
template <class T, int HD>
__device__ __forceinline__ void zero_rows(uint8_t *s_v, int r0, int r1) {
    for (int i = threadIdx.x; i < (r1 - r0) * (HD / 8); i += kAttnThreads)
        *reinterpret_cast<uint4 *>(T::frag(s_v, r0 + i / (HD / 8), i & 1, i % (HD / 8) >> 1)) = make_uint4(0, 0, 0, 0);
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Bounded wait for phase 0 of a copy barrier.
__device__ __forceinline__ bool attn_wait(uint64_t *bar) {
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
    for (uint32_t i = 0; i < (1u << 22); i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(b), "r"(0u)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Four 8x8 matrices of halves; lane l supplies the address of row l % 8 of matrix l / 8.  Plain: thread (g, t) gets
// elements [g][2t], [g][2t+1] of each matrix; .trans: elements [2t][g], [2t+1][g].
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void *row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(row)));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], const void *row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(row)));
}
// D += A(16x8, f16) * B(8x8, f16), f32 accumulate.  (Eight products a step: the bits of the tf32 instruction on the same values.  The step of
// sixteen rounds differently, and 32 layers carry a last bit on to 0.04 of the result.)
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(b));
}
// f16 pieces of two f32 values: hi = the top 11 significant bits, mid = the top 11 of what is left, times 2^11
__device__ __forceinline__ void f16_pieces(float x, float y, uint32_t &hi, uint32_t &mid) {
    const __half hx = __float2half_rz(x), hy = __float2half_rz(y);
    const __half2 h = __halves2half2(hx, hy), m = __halves2half2(__float2half_rz((x - __half2float(hx)) * 2048.0f), __float2half_rz((y - __half2float(hy)) * 2048.0f));
    hi = *reinterpret_cast<const uint32_t *>(&h);
    mid = *reinterpret_cast<const uint32_t *>(&m);
}
constexpr float kMid = 1.0f / 2048.0f;
// The f16 pieces of a scaled element that is not zero lose bits below 2^-12: its last bit is below 2^-35 then, the last bit of the second piece.
constexpr float kShort = 1.0f / 4096.0f;
// The pieces of one head's query by a warp: columns 2 * pair, 2 * pair + 1 of s_q (rows of QS halves); returns what a sum of products is
// to be multiplied by.  small: set where an element of this lane loses bits (or is zero: cheaper to ask, and rare).
template <int HD, int QS>
__device__ __forceinline__ float split_query(const float *qrow, __half *s_q, int pair, int lane, bool valid, bool &small) {
    constexpr int N = HD / 64;
    float2 v[N];
    float am = 0.f, least = INFINITY;
#pragma unroll
    for (int i = 0; i < N; i++) {
        v[i] = valid ? *reinterpret_cast<const float2 *>(qrow + i * 64 + lane * 2) : make_float2(0.f, 0.f);
        am = fmaxf(am, fmaxf(fabsf(v[i].x), fabsf(v[i].y)));
        least = fminf(least, fminf(fabsf(v[i].x), fabsf(v[i].y)));
    }
    am = warp_max(am);
    const int e = (int)(__float_as_uint(am) >> 23);
    const float f = __uint_as_float((uint32_t)min(268 - max(e, 1), 254) << 23);  // am * f is in [2^14, 2^15)
#pragma unroll
    for (int i = 0; i < N; i++) {
        uint32_t hi, mid;
        f16_pieces(v[i].x * f, v[i].y * f, hi, mid);
        *reinterpret_cast<uint32_t *>(s_q + (2 * pair) * QS + i * 64 + lane * 2) = hi;
        *reinterpret_cast<uint32_t *>(s_q + (2 * pair + 1) * QS + i * 64 + lane * 2) = mid;
    }
    small = small || (valid && least * f < kShort);
    return 1.0f / f;
}
// Scores of one head (f32, 128 keys, `keys` of them valid) -> this lane's four of exp(s - m), and m and l in ml.
__device__ __forceinline__ void tile_weights(const float *s_sc, int lane, int keys, float factor, float *ml, float (&v)[4]) {
    float m = -INFINITY;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        v[e] = lane + 32 * e < keys ? __fmul_rn(s_sc[lane + 32 * e], factor) : -INFINITY;
        m = fmaxf(m, v[e]);
    }
    m = warp_max(m);
    float l = 0.f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        v[e] = keys > 0 ? expf(v[e] - m) : 0.f;
        l += v[e];
    }
    l = warp_sum(l);
    if (lane == 0) ml[0] = m, ml[1] = l;
}
// The weights' pieces in columns 2 * pair, 2 * pair + 1 of s_p.  Returns whether a weight of this lane loses bits.
template <int PS>
__device__ __forceinline__ bool softmax_tile(const float *s_sc, __half *s_p, int pair, int lane, int keys, float factor, float *ml) {
    float v[4];
    tile_weights(s_sc, lane, keys, factor, ml, v);
    uint32_t least = 0xFFFFFFFFu;  // of the bits - 1: zero becomes the largest number
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float w = v[e] * 32768.0f;
        least = min(least, __float_as_uint(v[e]) - 1u);
        const __half hi = __float2half_rz(w);
        s_p[(2 * pair) * PS + lane + 32 * e] = hi;
        s_p[(2 * pair + 1) * PS + lane + 32 * e] = __float2half_rz((w - __half2float(hi)) * 2048.0f);
    }
    return least < __float_as_uint(kShort / 32768.0f) - 1u;
}
constexpr float kWeight = 1.0f / 32768.0f;
// The B words of one lane: column g8 of a group of eight, elements 2 t4, 2 t4 + 1 and 2 t4 + 8, 2 t4 + 9 from `k0` on
template <int S>
__device__ __forceinline__ void b_words(const __half *cols, int col, int k0, int t4, uint32_t &b0, uint32_t &b1) {
    const __half *p = cols + col * S + k0 + 2 * t4;
    b0 = *reinterpret_cast<const uint32_t *>(p);
    b1 = *reinterpret_cast<const uint32_t *>(p + 8);
}

// D += A(16x8, tf32) * B(8x8, tf32), f32 accumulate
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// tf32 pieces of an f32 value: piece 0 = its top 11 significant bits, piece 1 = the top 11 of what is left
__device__ __forceinline__ uint32_t tf32_piece(float v, int piece) {
    const uint32_t hi = __float_as_uint(v) & 0xFFFFE000u;
    return piece == 0 ? hi : (__float_as_uint(v - __uint_as_float(hi)) & 0xFFFFE000u);
}
// Two 16x8 tf32 fragments from the four matrices of an ldmatrix of halves.  The K index of the instruction is only a summation index: slot t takes
// element 2t of a group of 8 and slot t + 4 element 2t + 1, which is how ldmatrix hands out halves in pairs.
__device__ __forceinline__ void widen(const uint32_t (&r)[4], uint32_t (&a)[2][4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&r[i]));
        a[i >> 1][i & 1] = __float_as_uint(f.x);
        a[i >> 1][2 + (i & 1)] = __float_as_uint(f.y);
    }
}
// NT groups of four pairs from p0 on (at or past p_end: as the one before it) in one pass over the 16 x 16 fragments that `frag` loads: the pairs'
// f32 operands are at row(pair) + 16 step; sums(pair, v0, v1) gets rows g8 and g8 + 8.
template <int NT, int STEPS, class Frag, class Row, class Sums>
__device__ __forceinline__ void pairs_tf32(int p0, int p_end, const Frag &frag, const Row &row, const Sums &sums) {
    const int lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3, piece = g8 & 1;
    float acc[NT][4];
    const float *b[NT];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
        acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        b[nt] = row(min(p0 + nt * 4 + (g8 >> 1), p_end - 1)) + 2 * t4;
    }
#pragma unroll 4
    for (int j = 0; j < STEPS; j++) {
        uint32_t r[4], a[2][4];
        frag(r, j);
        widen(r, a);
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const float2 x = *reinterpret_cast<const float2 *>(b[nt] + j * 16), y = *reinterpret_cast<const float2 *>(b[nt] + j * 16 + 8);
            mma_tf32(acc[nt], a[0], tf32_piece(x.x, piece), tf32_piece(x.y, piece));
            mma_tf32(acc[nt], a[1], tf32_piece(y.x, piece), tf32_piece(y.y, piece));
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++)
        if (p0 + nt * 4 + t4 < p_end) sums(p0 + nt * 4 + t4, acc[nt][0] + acc[nt][1], acc[nt][2] + acc[nt][3]);
}
// A landed tile for the `pairs` (row, head) pairs of rows 0 .. pairs / G - 1, both products in tf32 pieces: the bits of the f16 form where that one
// loses none.  Row r sees keys0 + r keys of the tile; sc: [pair][kAttnTile], the scores, to be multiplied by f[pair]; rescore: an element of a query
// loses bits too, so the scores come again from q.  q, part_o, part_ml: of row 0 and head 0 of the group.
// A function of its own behind which the kernels return (few tiles need it), its arguments in registers: as a structure they lie in local memory, which
// has little L1 beside that much shared memory (1 us a tile).  Where every tile takes it: 32 sequences at 4097 keys, 32 heads / 8, 103 -> 121 us.
template <class T, int HD, int G, int P>
__device__ __noinline__ void tile_tf32(uint8_t *s_k, uint8_t *s_v, float *sc, const float *f, float (*ml)[2], const float *q, float *part_o, float *part_ml, int n_head,
                                       int n_splits, int pairs, int keys0, float scale, bool rescore) {
    constexpr int DG = HD / 16, KP = (kAttnThreads / 32) / DG, KEYS = kAttnTile / KP, NT = (P + 3) / 4, NT1 = (G + 3) / 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2;
    auto out_of = [&](int pair) { return ((size_t)(pair / G) * n_head + pair % G) * n_splits; };
    if (rescore) {  // scores of keys 16 warp .. 16 warp + 15
        const int arow = 16 * warp + (lane & 7) + ((lane >> 3) & 1) * 8;
        pairs_tf32<NT, HD / 16>(
            0, pairs, [&](uint32_t(&r)[4], int j) { ldsm4(r, T::frag(s_k, arow, lane >> 4, j)); }, [&](int p) { return q + ((size_t)(p / G) * n_head + p % G) * HD; },
            [&](int p, float v0, float v1) { sc[p * kAttnTile + 16 * warp + g8] = v0, sc[p * kAttnTile + 16 * warp + g8 + 8] = v1; });
        __syncthreads();
    }
    for (int p = warp; p < pairs; p += kAttnThreads / 32) {  // the weights in the scores' place
        float v[4];
        tile_weights(sc + p * kAttnTile, lane, min(kAttnTile, keys0 + p / G), rescore ? scale : f[p], ml[p], v);
#pragma unroll
        for (int e = 0; e < 4; e++) sc[p * kAttnTile + lane + 32 * e] = v[e];
    }
    __syncthreads();
    if (tid < pairs) part_ml[out_of(tid) * 2] = ml[tid][0], part_ml[out_of(tid) * 2 + 1] = ml[tid][1];
    // output dims 16 dg .. + 15 over this warp's share of the keys; a row at a time, last row first, where the rows see different keys: 0 must not
    // meet an infinity of a later token
    const int dg = warp % DG, kp = warp / DG, nr = pairs / G;
    const uint8_t *vrow = T::frag(s_v, kp * KEYS + (lane & 7) + (lane >> 4) * 8, (lane >> 3) & 1, dg);
    float *s_o = reinterpret_cast<float *>(s_k);  // KP > 1: [KP][G][HD], the key tile is dead
    auto values = [&](auto ntc, int first, int end) {
        pairs_tf32<decltype(ntc)::value, KEYS / 16>(
            first, end, [&](uint32_t(&r)[4], int j) { ldsm4_trans(r, vrow + j * 16 * T::kStride); }, [&](int p) { return sc + p * kAttnTile + kp * KEYS; },
            [&](int p, float v0, float v1) {
                float *o = (KP == 1 ? part_o + out_of(p) * HD : s_o + (kp * G + p) * HD) + 16 * dg + g8;
                o[0] = v0, o[8] = v1;
            });
    };
    if (P == G || keys0 >= kAttnTile) {
        values(std::integral_constant<int, NT>{}, 0, pairs);
    } else {
        for (int r = nr - 1; r >= 0 && keys0 + r > 0; r--) {
            if (r != nr - 1) {
                __syncthreads();  // the row after this one has been multiplied
                if (keys0 + r < kAttnTile && tid < HD / 8) *reinterpret_cast<uint4 *>(T::frag(s_v, keys0 + r, tid & 1, tid >> 1)) = make_uint4(0, 0, 0, 0);
                __syncthreads();
            }
            values(std::integral_constant<int, NT1>{}, r * G, r * G + G);
        }
    }
    if (KP > 1) {
        __syncthreads();
        for (int i = tid; i < G * HD; i += kAttnThreads) {
            float t = s_o[i];
#pragma unroll
            for (int w = 1; w < KP; w++) t += s_o[w * G * HD + i];
            part_o[out_of(i / HD) * HD + i % HD] = t;
        }
    }
}

constexpr int kAttnChunkPairs = 16;   // (query row, head) pairs of a chunk's tile
constexpr int kAttnPad = 8;  // halves behind a column of 64 or 128: the eight columns of a read start four banks apart

template <int HD, int G, bool BOXED>
__global__ void __launch_bounds__(kAttnThreads) attn_split_kernel(const float *q, const __half *k_cache,
                                                               const __half *v_cache, float *__restrict__ part_o,
                                                               float *__restrict__ part_ml, int rows, int n_head, int n_kv, int pos,
                                                               float scale, int n_splits, size_t seq_stride, uint32_t *__restrict__ status,
                                                               const int32_t *seq_pos, const int32_t *block_table,
                                                               int table_stride, int n_pages, const __grid_constant__ std::conditional_t<BOXED, AttnMaps, NoMaps> maps) {
    constexpr int CPR = HD * 2 / 16;           // 16-byte pieces per row
    constexpr int NT = (2 * G + 7) / 8;        // 8-column groups of the instruction: column c = head c / 2, piece c % 2
    constexpr int DG = HD / 16;                // 16-dim output groups
    constexpr int KP = (kAttnThreads / 32) / DG;  // warps per output group: they split the keys (1 for head_dim 128, 2 for 64)
    using T = std::conditional_t<BOXED, BoxedTile<HD>, PaddedTile<HD>>;
    extern __shared__ __align__(16) uint8_t dyn_smem[];
    uint8_t *s_k = align_tile<T>(dyn_smem), *s_v = s_k + T::kBytes;
    float(*s_o)[G][HD] = reinterpret_cast<float(*)[G][HD]>(s_k);  // KP x G x HD floats over the key tile (KP > 1 only)
    constexpr int QS = HD + kAttnPad, PS = kAttnTile + kAttnPad;
    __shared__ __align__(16) __half s_q[NT * 8 * QS];  // columns past 2 G are never stored
    __shared__ __align__(16) __half s_p[NT * 8 * PS];
    __shared__ __align__(16) float s_sc[G][kAttnTile];
    __shared__ float s_f[G];
    __shared__ float s_ml[G][2];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ int s_short[2];  // a weight, an element of a query loses bits
    static_assert(KP * G * HD * 4 <= T::kBytes, "the partial outputs reuse the key tile");
    static_assert(KP >= 1 && KP * DG == kAttnThreads / 32, "head_dim 64 or 128");
    const int split = blockIdx.x, kvh = blockIdx.y, qr = blockIdx.z;
    const int seq = qr / rows, ti = qr % rows;
    const int key0 = split * kAttnTile;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
    if (tid < 2) s_short[tid] = 0;
    if constexpr (BOXED) {
        init_bars<HD>(s_bar, maps);
        __syncthreads();
    }
    pdl_go();
    pdl_wait();
    // sequences at positions of their own (seq_pos, written by an earlier kernel or the host): `pos` is their maximum
    const int n_keys = (seq_pos ? max(0, min(seq_pos[seq], pos)) : pos) + ti + 1;
    const size_t out_idx = ((size_t)qr * n_head + (size_t)kvh * G) * n_splits + split;  // + g * n_splits
    if (key0 >= n_keys) {  // a tile beyond this row's causal end contributes nothing
        if (tid < G) {
            part_ml[(out_idx + (size_t)tid * n_splits) * 2] = -INFINITY;
            part_ml[(out_idx + (size_t)tid * n_splits) * 2 + 1] = 0.f;
        }
        return;
    }
    // contiguous caches: the sequence's own rows; paged: the tile is one page of the pool (a page holds a tile's 128 rows)
    const size_t kv_row = (size_t)n_kv * HD;
    const int page = block_table ? min(max(block_table[(size_t)seq * table_stride + split], 0), n_pages - 1) : 0;
    const int tile_keys = min(kAttnTile, n_keys - key0);
    // Two ways to fetch the tile.  BOXED (more than two waves of CTAs: a batch of sequences): tensor copies of 64 dims, so that
    // a tile costs its warps next to nothing; keys and values complete on separate barriers.  Otherwise (a single wave of
    // CTAs, where the latency of the first byte is what counts): 16-byte cp.async, consecutive threads taking consecutive
    // pieces of a row.
    if constexpr (BOXED) {
        fetch_tile<HD>(maps, s_k, s_v, s_bar, kvh, block_table ? page * kAttnTile : key0, block_table ? 0 : seq, tile_keys);
    } else {
        const size_t tile_off = (size_t)kvh * HD + (block_table ? (size_t)page * kAttnTile * kv_row : (size_t)seq * seq_stride + (size_t)key0 * kv_row);
        for (int i = tid; i < tile_keys * CPR; i += kAttnThreads) {
            const int key = i / CPR, c = i % CPR;
            cp_async16(s_k + key * T::kStride + c * 16, k_cache + tile_off + (size_t)key * kv_row + c * 8);
        }
        cp_async_commit();
        for (int i = tid; i < tile_keys * CPR; i += kAttnThreads) {
            const int key = i / CPR, c = i % CPR;
            cp_async16(s_v + key * T::kStride + c * 16, v_cache + tile_off + (size_t)key * kv_row + c * 8);
        }
        cp_async_commit();
    }
    zero_rows<T, HD>(s_v, BOXED ? boxed_rows(tile_keys) : tile_keys, kAttnTile);
    const float *qrow = q + ((size_t)qr * n_head + (size_t)kvh * G) * HD;
    bool small = false;
    for (int g = warp; g < NT * 4; g += kAttnThreads / 32) {
        const float f = split_query<HD, QS>(qrow + (size_t)g * HD, s_q, g, lane, g < G, small);
        if (lane == 0 && g < G) s_f[g] = f * scale;
    }
    // the keys have landed; q is staged.  (BOXED: a bounded wait; if it runs out, the CTA
    // records it and leaves after the wait for the values has had its own limit, so that no copy can land in shared
    // memory that is no longer this CTA's.)
    if (BOXED) {
        const bool k_ok = attn_wait(&s_bar[0]);
        if (!__syncthreads_and(k_ok)) {
            attn_wait(&s_bar[1]);
            if (tid == 0) atomicExch(status, 12u);
            return;
        }
    } else {
        cp_async_wait<1>();
        __syncthreads();
    }
    // ---- phase 1: scores of keys 16 warp .. 16 warp + 15
    {
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        // ldmatrix rows: matrices 0 / 1 = keys 0..7 / 8..15 at dims d0.., matrices 2 / 3 = the same keys at dims d0 + 8..
        const int arow = 16 * warp + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int j = 0; j < HD / 16; j++) {
            uint32_t r[4];
            ldsm4(r, T::frag(s_k, arow, lane >> 4, j));
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                uint32_t b0, b1;
                b_words<QS>(s_q, nt * 8 + g8, j * 16, t4, b0, b1);
                mma_f16(acc[nt], r[0], r[1], b0);
                mma_f16(acc[nt], r[2], r[3], b1);
            }
        }
        // columns 2 t4, 2 t4 + 1 of group nt = the two pieces of head 4 nt + t4; rows g8 and g8 + 8 of the warp's keys
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int head = nt * 4 + t4;
            if (head < G) {
                s_sc[head][16 * warp + g8] = fmaf(acc[nt][1], kMid, acc[nt][0]);
                s_sc[head][16 * warp + g8 + 8] = fmaf(acc[nt][3], kMid, acc[nt][2]);
            }
        }
    }
    // the values have landed; scores complete, key tile no longer read
    if (BOXED) {
        const bool v_ok = attn_wait(&s_bar[1]);
        if (!__syncthreads_and(v_ok)) {
            if (tid == 0) atomicExch(status, 12u);
            return;
        }
    } else {
        cp_async_wait<0>();
        __syncthreads();
    }
    // ---- phase 2
    if (BOXED) zero_rows<T, HD>(s_v, tile_keys, boxed_rows(tile_keys));
    if (small) s_short[1] = 1;
    small = false;
    for (int g = warp; g < G; g += kAttnThreads / 32) small = softmax_tile<PS>(s_sc[g], s_p, g, lane, tile_keys, s_f[g], s_ml[g]) || small;
    if (small) s_short[0] = 1;
    __syncthreads();
    if (s_short[0] || s_short[1]) {
        tile_tf32<T, HD, G, G>(
            s_k, s_v, s_sc[0], s_f, s_ml, qrow, part_o + out_idx * HD, part_ml + out_idx * 2, n_head, n_splits, G, tile_keys, scale, s_short[1] != 0);
        return;
    }
    // ---- phase 3: output dims 16 dg .. + 15 over this warp's share of the keys
    {
        const int dg = warp % DG, kp = warp / DG;
        constexpr int KEYS = kAttnTile / KP;
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        // ldmatrix.trans rows: matrices 0 / 1 = keys 0..7 at dims 0..7 / 8..15 of the group, matrices 2 / 3 = keys 8..15
        const uint8_t *vrow = T::frag(s_v, kp * KEYS + (lane & 7) + (lane >> 4) * 8, (lane >> 3) & 1, dg);
#pragma unroll
        for (int s16 = 0; s16 < KEYS / 16; s16++) {
            uint32_t r[4];
            ldsm4_trans(r, vrow + s16 * 16 * T::kStride);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                uint32_t b0, b1;
                b_words<PS>(s_p, nt * 8 + g8, kp * KEYS + s16 * 16, t4, b0, b1);
                mma_f16(acc[nt], r[0], r[1], b0);
                mma_f16(acc[nt], r[2], r[3], b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int head = nt * 4 + t4;
            if (head < G) {
                const float o0 = fmaf(acc[nt][1], kMid, acc[nt][0]) * kWeight, o1 = fmaf(acc[nt][3], kMid, acc[nt][2]) * kWeight;  // dims 16 dg + g8, + 8
                if (KP == 1) {
                    float *po = part_o + (out_idx + (size_t)head * n_splits) * HD + 16 * dg + g8;
                    po[0] = o0;
                    po[8] = o1;
                } else {
                    s_o[kp][head][16 * dg + g8] = o0;
                    s_o[kp][head][16 * dg + g8 + 8] = o1;
                }
            }
        }
    }
    if (KP > 1) {
        __syncthreads();
        for (int i = tid; i < G * HD; i += kAttnThreads) {
            const int g = i / HD, d = i % HD;
            float t = s_o[0][g][d];
#pragma unroll
            for (int w = 1; w < KP; w++) t += s_o[w][g][d];
            part_o[(out_idx + (size_t)g * n_splits) * HD + d] = t;
        }
    }
    if (tid < G) {
        part_ml[(out_idx + (size_t)tid * n_splits) * 2] = s_ml[tid][0];
        part_ml[(out_idx + (size_t)tid * n_splits) * 2 + 1] = s_ml[tid][1];
    }
}

// The same tile for 16 / G consecutive query rows of one sequence (a prompt chunk), head_dim 128: 16 (row, head) pairs are 32
// columns of the matrix instruction, so a key or value fragment is loaded once for all of them; the arithmetic of a
// column, and so every bit, is that of attn_split_kernel.  Where a tile ends inside the rows' causal edge and a value there is infinite or
// NaN, the values are multiplied row by row, last row first: each row sees one key fewer, and that key's values are zeroed, so that the
// matrix unit multiplies 0 (not a later token's infinity) by its weight 0.
// Measured (us a call with the merge, 113 rows at position 384, 32 heads / 8): in tf32 pieces with the edge always row by row and eight warps a merged
// block 46, now 29 (all eight steps of a product unrolled 31.5).
template <int G, bool BOXED>
__global__ void __launch_bounds__(kAttnThreads) attn_chunk_kernel(const float *q, const __half *k_cache,
                                                                  const __half *v_cache, float *__restrict__ part_o,
                                                                  float *__restrict__ part_ml, int rows, int n_head, int n_kv, int pos, float scale,
                                                                  int n_splits, size_t seq_stride, uint32_t *__restrict__ status,
                                                                  const int32_t *seq_pos, const int32_t *block_table,
                                                                  int table_stride, int n_pages, const __grid_constant__ std::conditional_t<BOXED, AttnMaps, NoMaps> maps) {
    constexpr int HD = 128, P = kAttnChunkPairs, S = HD + kAttnPad, R = P / G, CPR = HD * 2 / 16, NT = 2 * P / 8, NT1 = (2 * G + 7) / 8;
    static_assert(kAttnTile == HD, "one stride for queries and weights");
    using T = std::conditional_t<BOXED, BoxedTile<HD>, PaddedTile<HD>>;
    static_assert(kAttnThreads / 32 == HD / 16, "a warp owns 16 output dims");
    extern __shared__ __align__(16) uint8_t dyn_smem[];
    uint8_t *s_k = align_tile<T>(dyn_smem), *s_v = s_k + T::kBytes;
    __half *s_q = reinterpret_cast<__half *>(s_v + T::kBytes);        // [2 P][S]: the queries' pieces
    __half *s_p = s_q + 2 * P * S;                                         // [2 P][S]: the weights' pieces
    float(*s_sc)[kAttnTile] = reinterpret_cast<float(*)[kAttnTile]>(s_p + 2 * P * S);  // [P][128]
    __shared__ float s_f[P];
    __shared__ float s_ml[P][2];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ int s_short[2];  // a weight, an element of a query loses bits
    const int row_blocks = (rows + R - 1) / R;
    const int split = blockIdx.x, kvh = blockIdx.y, seq = blockIdx.z / row_blocks, ti0 = (blockIdx.z % row_blocks) * R, nr = min(R, rows - ti0);
    const int key0 = split * kAttnTile;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
    if (tid < 2) s_short[tid] = 0;
    if constexpr (BOXED) {
        init_bars<HD>(s_bar, maps);
        __syncthreads();
    }
    pdl_go();
    pdl_wait();
    const int base = (seq_pos ? max(0, min(seq_pos[seq], pos)) : pos) + ti0 + 1 - key0;  // keys of this tile that row r sees: base + r
    auto out_of = [&](int pair) {
        return (((size_t)seq * rows + ti0 + pair / G) * n_head + (size_t)kvh * G + pair % G) * n_splits + split;
    };
    const int tile_keys = min(kAttnTile, base + nr - 1);
    if (tile_keys <= 0) {  // a tile beyond every row's causal end contributes nothing
        if (tid < nr * G) part_ml[out_of(tid) * 2] = -INFINITY, part_ml[out_of(tid) * 2 + 1] = 0.f;
        return;
    }
    const int page = block_table ? min(max(block_table[(size_t)seq * table_stride + split], 0), n_pages - 1) : 0;
    const size_t kv_row = (size_t)n_kv * HD;
    if constexpr (BOXED) {
        fetch_tile<HD>(maps, s_k, s_v, s_bar, kvh, block_table ? page * kAttnTile : key0, block_table ? 0 : seq, tile_keys);
        zero_rows<T, HD>(s_v, boxed_rows(tile_keys), kAttnTile);
    } else {
        // A bulk copy for a row: thread r < 128 the key row r, thread 128 + r the value row r, or zeroes where the row lies past the end.  (Barriers made ready apart
        // and rows zeroed by all threads together: 8 / 8 heads, 64 rows at 384 8.24 -> 8.36 us, with an infinite last value 16.1 -> 16.5.)
        const int which = tid >> 7, r = tid & (kAttnTile - 1);
        if (tid == 0) {
            init_bars<64>(s_bar);
#pragma unroll
            for (int i = 0; i < 2; i++)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(s_bar + i)),
                             "r"((uint32_t)(tile_keys * HD * 2))
                             : "memory");
        }
        __syncthreads();  // the barriers are armed before any copy can complete
        if (r < tile_keys) {
            const __half *src = (which ? v_cache : k_cache) + (size_t)kvh * HD + (block_table ? (size_t)page * kAttnTile * kv_row : (size_t)seq * seq_stride + (size_t)key0 * kv_row) + (size_t)r * kv_row;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(T::frag(which ? s_v : s_k, r, 0, 0))),
                         "l"(src), "r"((uint32_t)(HD * 2)), "r"((uint32_t)__cvta_generic_to_shared(s_bar + which))
                         : "memory");
        } else if (which) {
#pragma unroll
            for (int c = 0; c < CPR; c++) *reinterpret_cast<uint4 *>(s_v + r * T::kStride + c * 16) = make_uint4(0, 0, 0, 0);
        }
    }
    const float *qrow = q + (((size_t)seq * rows + ti0) * n_head + (size_t)kvh * G) * HD;
    bool small = false;
    for (int pair = warp; pair < P; pair += kAttnThreads / 32) {
        const int r = pair / G;
        const float f = split_query<HD, S>(qrow + ((size_t)r * n_head + pair % G) * HD, s_q, pair, lane, r < nr, small);
        if (lane == 0) s_f[pair] = f * scale;
    }
    // (bounded waits; a CTA that gives up leaves after both copies have had their limit)
    const bool k_ok = attn_wait(&s_bar[0]);
    if (!__syncthreads_and(k_ok)) {
        attn_wait(&s_bar[1]);
        if (tid == 0) atomicExch(status, 12u);
        return;
    }
    // ---- phase 1: scores of keys 16 warp .. 16 warp + 15 for every pair
    {
        float acc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
        const int arow = 16 * warp + (lane & 7) + ((lane >> 3) & 1) * 8;
#pragma unroll 2
        for (int j = 0; j < HD / 16; j++) {
            uint32_t r[4];
            ldsm4(r, T::frag(s_k, arow, lane >> 4, j));
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                uint32_t b0, b1;
                b_words<S>(s_q, nt * 8 + g8, j * 16, t4, b0, b1);
                mma_f16(acc[nt], r[0], r[1], b0);
                mma_f16(acc[nt], r[2], r[3], b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            s_sc[nt * 4 + t4][16 * warp + g8] = fmaf(acc[nt][1], kMid, acc[nt][0]);
            s_sc[nt * 4 + t4][16 * warp + g8 + 8] = fmaf(acc[nt][3], kMid, acc[nt][2]);
        }
    }
    const bool v_ok = attn_wait(&s_bar[1]);
    if (!__syncthreads_and(v_ok)) {
        if (tid == 0) atomicExch(status, 12u);
        return;
    }
    // ---- phase 2
    if (BOXED) zero_rows<T, HD>(s_v, tile_keys, boxed_rows(tile_keys));
    if (small) s_short[1] = 1;
    small = false;
    for (int p = warp; p < P; p += kAttnThreads / 32)
        small = softmax_tile<S>(s_sc[p], s_p, p, lane, p / G < nr ? min(kAttnTile, base + p / G) : 0, s_f[p], s_ml[p]) || small;
    if (small) s_short[0] = 1;
    // The rows see different numbers of keys where the tile ends inside their causal edge: a key that one of them does not see has weight 0
    // there, which must not meet an infinity of a later token.
    bool apart = false;
    if (base < kAttnTile)
        for (int i = tid; i < (min(base + nr - 1, kAttnTile) - max(base, 0)) * HD / 2; i += kAttnThreads) {
            const int c = i % (HD / 2) >> 2;  // of four words
            const uint32_t w = *reinterpret_cast<const uint32_t *>(T::frag(s_v, max(base, 0) + i / (HD / 2), c & 1, c >> 1) + (i & 3) * 4);
            apart = apart || (w & 0x7C00u) == 0x7C00u || (w & 0x7C000000u) == 0x7C000000u;
        }
    apart = __syncthreads_or(apart);
    if (s_short[0] || s_short[1]) {
        tile_tf32<T, HD, G, P>(
            s_k, s_v, s_sc[0], s_f, s_ml, qrow, part_o + out_of(0) * HD, part_ml + out_of(0) * 2, n_head, n_splits, nr * G, base, scale, s_short[1] != 0);
        return;
    }
    // ---- phase 3: output dims 16 warp .. + 15
    const uint8_t *vrow = T::frag(s_v, (lane & 7) + (lane >> 4) * 8, (lane >> 3) & 1, warp);
    // NTC groups of four pairs from pair p0 on; pairs at or past p1 are computed for nothing and not stored
    auto values = [&](auto ntc, int p0, int p1) {
        constexpr int NTC = decltype(ntc)::value;
        float acc[NTC][4];
#pragma unroll
        for (int nt = 0; nt < NTC; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll 2
        for (int s16 = 0; s16 < kAttnTile / 16; s16++) {
            uint32_t r[4];
            ldsm4_trans(r, vrow + s16 * 16 * T::kStride);
#pragma unroll
            for (int nt = 0; nt < NTC; nt++) {
                uint32_t b0, b1;
                b_words<S>(s_p, min(2 * p0 + nt * 8 + g8, 2 * P - 1), s16 * 16, t4, b0, b1);
                mma_f16(acc[nt], r[0], r[1], b0);
                mma_f16(acc[nt], r[2], r[3], b1);
            }
        }
#pragma unroll
        for (int nt = 0; nt < NTC; nt++) {
            const int pair = p0 + nt * 4 + t4;
            if (pair < p1) {
                float *po = part_o + out_of(pair) * HD + 16 * warp + g8;
                po[0] = fmaf(acc[nt][1], kMid, acc[nt][0]) * kWeight;
                po[8] = fmaf(acc[nt][3], kMid, acc[nt][2]) * kWeight;
            }
        }
    };
    if (!apart) {
        values(std::integral_constant<int, NT>{}, 0, nr * G);
    } else {
#pragma unroll 1
        for (int r = nr - 1; r >= 0 && base + r > 0; r--) {
            if (r != nr - 1) {
                __syncthreads();  // the row after this one has been multiplied
                if (base + r < kAttnTile && tid < CPR) *reinterpret_cast<uint4 *>(T::frag(s_v, base + r, tid & 1, tid >> 1)) = make_uint4(0, 0, 0, 0);
                __syncthreads();
            }
            values(std::integral_constant<int, NT1>{}, r * G, r * G + G);
        }
    }
    if (tid < nr * G) part_ml[out_of(tid) * 2] = s_ml[tid][0], part_ml[out_of(tid) * 2 + 1] = s_ml[tid][1];
}

// CTA = (query row, head), thread = output dim: merges the tiles' (m, l, o).
__global__ void attn_combine_kernel(const float *part_o, const float *part_ml, float *__restrict__ dst,
                                    int head_dim, int n_splits) {
    pdl_go();
    pdl_wait();
    const size_t rh = blockIdx.x;
    const float *ml = part_ml + rh * n_splits * 2;
    float m = -INFINITY;
    for (int s = 0; s < n_splits; s++) m = fmaxf(m, ml[2 * s]);
    float l = 0.f, o = 0.f;
    for (int s = 0; s < n_splits; s++) {
        const float ls = ml[2 * s + 1];
        if (ls == 0.f) continue;
        const float wgt = expf(ml[2 * s] - m);
        l += wgt * ls;
        o = fmaf(wgt, part_o[(rh * n_splits + s) * head_dim + threadIdx.x], o);
    }
    dst[rh * head_dim + threadIdx.x] = o / l;
}

// ---------------------------------------------------------------------------------------------- elementwise
__global__ void __launch_bounds__(256) gated_silu_kernel(const float *gate, const float *up,
                                                         float *__restrict__ dst, size_t n) {
    pdl_go();
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float g = gate[i];
        dst[i] = silu_mul(g, up[i]);
    }
}

__global__ void __launch_bounds__(256) add_kernel(const float *a, const float *b, float *__restrict__ dst, size_t n) {
    pdl_go();
    pdl_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] = a[i] + b[i];
}

// Strict `>` with the lowest index on ties, per row.  Stage 1: CTA (chunk, row) -> best of its chunk;
// stage 2: one CTA per row over the chunk winners.
__device__ __forceinline__ void argmax_merge(float &bv, uint32_t &bi, float v, uint32_t i) {
    if (v > bv || (v == bv && i < bi)) bv = v, bi = i;
}
__device__ __forceinline__ void argmax_block(float bv, uint32_t bi, float *s_v, uint32_t *s_i, float *ov, uint32_t *oi) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, bv, o);
        const uint32_t i = __shfl_xor_sync(0xffffffffu, bi, o);
        argmax_merge(bv, bi, v, i);
    }
    if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = bv, s_i[threadIdx.x >> 5] = bi;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int nw = (blockDim.x + 31) / 32;
        bv = threadIdx.x < nw ? s_v[threadIdx.x] : -INFINITY;
        bi = threadIdx.x < nw ? s_i[threadIdx.x] : 0xffffffffu;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float v = __shfl_xor_sync(0xffffffffu, bv, o);
            const uint32_t i = __shfl_xor_sync(0xffffffffu, bi, o);
            argmax_merge(bv, bi, v, i);
        }
        if (threadIdx.x == 0) *ov = bv, *oi = bi;
    }
}

__global__ void __launch_bounds__(256) argmax_stage1_kernel(const float *x, float *__restrict__ cand_v,
                                                            uint32_t *__restrict__ cand_i, uint32_t n, uint32_t chunk) {
    __shared__ float s_v[32];
    __shared__ uint32_t s_i[32];
    pdl_go();
    pdl_wait();
    const uint32_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
    const float *row = x + (size_t)blockIdx.y * n;
    float bv = -INFINITY;
    uint32_t bi = 0xffffffffu;
    for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) argmax_merge(bv, bi, row[i], i);
    argmax_block(bv, bi, s_v, s_i, cand_v + (size_t)blockIdx.y * gridDim.x + blockIdx.x, cand_i + (size_t)blockIdx.y * gridDim.x + blockIdx.x);
}

__global__ void __launch_bounds__(256) argmax_stage2_kernel(const float *cand_v, const uint32_t *cand_i,
                                                            uint32_t *__restrict__ dst, uint32_t n_chunks) {
    __shared__ float s_v[32];
    __shared__ uint32_t s_i[32];
    __shared__ float s_bv;
    __shared__ uint32_t s_bi;
    pdl_go();
    pdl_wait();
    float bv = -INFINITY;
    uint32_t bi = 0xffffffffu;
    for (uint32_t c = threadIdx.x; c < n_chunks; c += blockDim.x)
        argmax_merge(bv, bi, cand_v[(size_t)blockIdx.x * n_chunks + c], cand_i[(size_t)blockIdx.x * n_chunks + c]);
    argmax_block(bv, bi, s_v, s_i, &s_bv, &s_bi);
    __syncthreads();
    // a row with no value above -inf (all -inf or NaN) answers index 0, like the reference's scan
    if (threadIdx.x == 0) dst[blockIdx.x] = s_bi == 0xffffffffu ? 0u : s_bi;
}

// ---------------------------------------------------------------------------------------------- producers that emit int8
// The activation quantiser's arithmetic for one 256-element block held by one warp (lane l owns elements 4l..4l+3
// and 128+4l..128+4l+3): d = amax / 127, id = d > 0 ? 1/d : 0, q = clamp(roundf(x * id), -127, 127), plus the
// per-32 and per-16 code sums (crates/infr-cpu/src/quant.rs:27-58).  Same operations in the same order as
// quantize_q8_kernel<256>, so a producer that ends with this emits the bits the separate quantiser would.
__device__ __forceinline__ float q8_amax4(float4 v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))); }
__device__ __forceinline__ void quantize_block256(const float4 v[2], int lane, size_t row, int k, int chunk, int8_t *__restrict__ qs,
                                                  float *__restrict__ d, int32_t *__restrict__ sums, int32_t *__restrict__ sums16) {
    float m = fmaxf(q8_amax4(v[0]), q8_amax4(v[1]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float dd = m / 127.0f;
    const float id = dd > 0.0f ? 1.0f / dd : 0.0f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int e = chunk * 256 + h * 128 + lane * 4;
        const uint32_t packed = q8_codes4(v[h], id);
        int sm = q8_sum4(packed);
        sm += __shfl_xor_sync(0xffffffffu, sm, 1);
        sm += __shfl_xor_sync(0xffffffffu, sm, 2);
        const int s16 = sm;
        sm += __shfl_xor_sync(0xffffffffu, sm, 4);
        *reinterpret_cast<uint32_t *>(qs + row * k + e) = packed;
        if (sums16 && (lane & 3) == 0) sums16[row * (k / 16) + e / 16] = s16;
        if ((lane & 7) == 0) sums[row * (k / 32) + e / 32] = sm;
    }
    if (lane == 0) d[row * (k / 256) + chunk] = dd;
}

// RMSNorm (rms_norm_row) whose output goes straight to int8.  With Q8 false the scaled row is stored as f32 to dst instead.
template <bool ADD, bool Q8>
__global__ void __launch_bounds__(1024) rms_norm_q8_kernel(const float *a, const float *b, float *sum_dst, const float *__restrict__ w, int dim,
                                                           float eps, float *__restrict__ dst, int8_t *__restrict__ qs, float *__restrict__ d,
                                                           int32_t *__restrict__ sums, int32_t *__restrict__ sums16) {
    __shared__ float s_part[32];
    const int lane = threadIdx.x & 31;
    rms_norm_row<ADD>(a, b, sum_dst, w, dim, eps, blockIdx.x, s_part, [&](int chunk, const float4 (&v)[2]) {
        if (Q8) {
            quantize_block256(v, lane, blockIdx.x, dim, chunk, qs, d, sums, sums16);
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) *reinterpret_cast<float4 *>(dst + (size_t)blockIdx.x * dim + chunk * 256 + h * 128 + lane * 4) = v[h];
        }
    });
}

// The consumer of a pushed row-parallel GEMV (GemvPush): row = a + sum over ranks of the partial results that the
// ranks' GEMV epilogues stored into this rank's staging, summed in rank order from zero (the order of the stand-alone
// all-reduce, so both forms give the same bits), written to sum_dst, then RMSNorm and the quantiser.  Every staged word
// carries its value and the exchange's sequence number: a thread polls, bounded, the four words of each rank that it
// is about to add, so nothing waits for data it does not read.  A thread whose poll runs out adds nothing and raises
// the status word.  The grid's last CTA opens the next exchange.  One CTA per row, dim % 256 == 0.
__device__ __forceinline__ void ld_words2(const unsigned long long *p, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__global__ void __launch_bounds__(1024) rms_norm_q8_pull_kernel(const float *a, float *sum_dst, const float *__restrict__ w, int dim, float eps,
                                                                int8_t *__restrict__ qs, float *__restrict__ d, int32_t *__restrict__ sums,
                                                                int32_t *__restrict__ sums16, PullArgs pull) {
    __shared__ float s_part[32];
    pdl_go();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, chunks = dim / 256;
    const bool in_regs = chunks <= nw;
    // the norm weights do not depend on the previous kernel: fetch them before waiting for it
    float4 g[2];
    if (in_regs && warp < chunks) {
#pragma unroll
        for (int h = 0; h < 2; h++) g[h] = *reinterpret_cast<const float4 *>(w + warp * 256 + h * 128 + lane * 4);
    }
    pdl_wait();
    const uint32_t done = *reinterpret_cast<volatile uint32_t *>(pull.ctrl);
    const uint32_t par = done & 1u, want = done + 1u;
    const size_t base = (size_t)blockIdx.x * dim;
    float4 x[2];
    float ss = 0.f;
    for (int chunk = warp; chunk < chunks; chunk += nw) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = chunk * 256 + h * 128 + lane * 4;
            float4 v = *reinterpret_cast<const float4 *>(a + base + e);  // the residual row does not depend on the peers
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            bool all = true;
            for (int r = 0; r < pull.world; r++) {
                const unsigned long long *src = pull.stage + ((size_t)par * pull.world + r) * pull.cap + base + e;
                unsigned long long w0, w1, w2, w3;
                uint32_t it = 0;
                bool ok;
                do {
                    ld_words2(src, w0, w1);
                    ld_words2(src + 2, w2, w3);
                    ok = (uint32_t)(w0 >> 32) == want && (uint32_t)(w1 >> 32) == want && (uint32_t)(w2 >> 32) == want && (uint32_t)(w3 >> 32) == want;
                } while (!ok && ++it < pull.spin);
                all = all && ok;
                acc.x += __uint_as_float((uint32_t)w0), acc.y += __uint_as_float((uint32_t)w1);
                acc.z += __uint_as_float((uint32_t)w2), acc.w += __uint_as_float((uint32_t)w3);
            }
            if (all)
                v.x += acc.x, v.y += acc.y, v.z += acc.z, v.w += acc.w;
            else
                atomicExch(pull.status, 11u);
            *reinterpret_cast<float4 *>(sum_dst + base + e) = v;
            ss = __fadd_rn(ss, sumsq4(v));
            x[h] = v;
        }
    }
    ss = warp_sum(ss);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    const float s = 1.0f / sqrtf(warp_sum(lane < nw ? s_part[lane] : 0.f) / (float)dim + eps);
    for (int chunk = warp; chunk < chunks; chunk += nw) {
        float4 v[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = chunk * 256 + h * 128 + lane * 4;
            if (!in_regs) {
                x[h] = *reinterpret_cast<const float4 *>(sum_dst + base + e);  // re-read by the warp that wrote it
                g[h] = *reinterpret_cast<const float4 *>(w + e);
            }
            v[h] = make_float4(x[h].x * s * g[h].x, x[h].y * s * g[h].y, x[h].z * s * g[h].z, x[h].w * s * g[h].w);
        }
        quantize_block256(v, lane, blockIdx.x, dim, chunk, qs, d, sums, sums16);
    }
    // every CTA has read the count and its words: the last one opens the next exchange
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(pull.ctrl + 1, 1u) == gridDim.x - 1) {
            pull.ctrl[1] = 0;
            __threadfence();
            *reinterpret_cast<volatile uint32_t *>(pull.ctrl) = done + 1u;
        }
    }
}

// silu(gate) * up straight to int8: warp = (row, 256-element block); nff % 256 == 0.
__global__ void __launch_bounds__(256) gated_silu_q8_kernel(const float *gate, const float *up, int rows, int nff,
                                                            int8_t *__restrict__ qs, float *__restrict__ d, int32_t *__restrict__ sums,
                                                            int32_t *__restrict__ sums16) {
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31, cpr = nff / 256;
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wg >= (long long)rows * cpr) return;
    const int row = (int)(wg / cpr), chunk = (int)(wg % cpr);
    float4 v[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const size_t e = (size_t)row * nff + chunk * 256 + h * 128 + lane * 4;
        const float4 g = *reinterpret_cast<const float4 *>(gate + e), u = *reinterpret_cast<const float4 *>(up + e);
        v[h] = make_float4(silu_mul(g.x, u.x), silu_mul(g.y, u.y), silu_mul(g.z, u.z), silu_mul(g.w, u.w));
    }
    quantize_block256(v, lane, (size_t)row, nff, chunk, qs, d, sums, sums16);
}

// The merge of the key tiles with the result quantised in place of an f32 store.  CTA = (query row, 256 outputs),
// 8 warps: warp h < heads-per-block first turns head h's tile maxima into weights exp(m_s - M) in shared memory,
// then warp w accumulates tiles w, w + 8, ... for the block's 256 outputs (lane = 2 x 4 dims), the eight partial
// sums meet in shared memory and warp 0 normalises and quantises.
// With Q8 false the same sums are stored as f32 instead, so the two forms agree bit for bit.
constexpr int kCombineMaxSplits = 512;
// AHEAD (few rows): a warp's first tiles are on their way while the weights are formed, one round trip to L2 where the loads came one after
// the other (one row, 33 tiles: 5.2 -> 4.1 us; 32 rows, whose registers it costs: 8.2 -> 10).
template <bool Q8, bool AHEAD>
__global__ void __launch_bounds__(256, AHEAD ? 1 : 4) attn_combine_wide_kernel(const float *part_o, const float *part_ml, int n_head,
                                                                int head_dim, int n_splits, float *__restrict__ dst, int8_t *__restrict__ qs,
                                                                float *__restrict__ d, int32_t *__restrict__ sums, int32_t *__restrict__ sums16) {
    __shared__ float s_w[4][kCombineMaxSplits];
    __shared__ float s_l[4];
    __shared__ int s_n[4];
    __shared__ __align__(16) float s_acc[8][256];
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = n_head * head_dim, cpr = k / 256;
    const int row = blockIdx.x / cpr, chunk = blockIdx.x % cpr;
    const int heads = 256 / head_dim, head0 = chunk * heads;
    constexpr int kAhead = AHEAD ? 4 : 0;
    float4 p[2][kAhead + 1];
    const float *po[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int e = h * 128 + lane * 4;
        po[h] = part_o + ((size_t)row * n_head + head0 + e / head_dim) * n_splits * head_dim + e % head_dim;
#pragma unroll
        for (int j = 0; j < kAhead; j++)
            if (warp + 8 * j < n_splits) p[h][j] = *reinterpret_cast<const float4 *>(po[h] + (size_t)(warp + 8 * j) * head_dim);
    }
    if (warp < heads) {
        const float2 *ml = reinterpret_cast<const float2 *>(part_ml) + ((size_t)row * n_head + head0 + warp) * n_splits;
        const float2 none = make_float2(-INFINITY, 0.f);
        const float2 ml0 = lane < n_splits ? ml[lane] : none, ml1 = lane + 32 < n_splits ? ml[lane + 32] : none;
        float m = fmaxf(ml0.x, ml1.x);
        for (int s = lane + 64; s < n_splits; s += 32) m = fmaxf(m, ml[s].x);
        m = warp_max(m);
        float l = 0.f;
        int n = 0;
        for (int s = lane; s < n_splits; s += 32) {
            const float2 v = s < 32 ? ml0 : s < 64 ? ml1 : ml[s];
            if (v.y == 0.f) break;  // past the row's causal end, as all tiles after it (a tile with keys has l >= 1, or NaN)
            const float wgt = expf(v.x - m);
            s_w[warp][s] = wgt;
            l += wgt * v.y;
            n = s + 1;
        }
        l = warp_sum(l);
        n = __reduce_max_sync(0xffffffffu, n);
        if (lane == 0) s_l[warp] = l, s_n[warp] = n;
    }
    __syncthreads();
    float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    auto add = [&](float4 &t, float wgt, float4 v) {
        t.x = fmaf(wgt, v.x, t.x), t.y = fmaf(wgt, v.y, t.y), t.z = fmaf(wgt, v.z, t.z), t.w = fmaf(wgt, v.w, t.w);
    };
    // (nobody writes the sums of the tiles past the causal end: what an earlier op left there may read as NaN)
    const int hh[2] = {lane * 4 / head_dim, (128 + lane * 4) / head_dim}, n[2] = {s_n[hh[0]], s_n[hh[1]]};
#pragma unroll
    for (int j = 0; j < kAhead; j++)
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (warp + 8 * j < n[h]) add(acc[h], s_w[hh[h]][warp + 8 * j], p[h][j]);
    // (Both halves' loads together, one round trip where there were two; without AHEAD with room for eight of them, four CTAs an SM.  us a call, 32 heads / 8 at
    // 4097 keys, before / after: 4 sequences 19.2 / 18.6, 16 51.2 / 50.1, 32 92.0 / 91.4.)
#pragma unroll 4
    for (int s = warp + 8 * kAhead; s < max(n[0], n[1]); s += 8)
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (s < n[h]) add(acc[h], s_w[hh[h]][s], *reinterpret_cast<const float4 *>(po[h] + (size_t)s * head_dim));
#pragma unroll
    for (int h = 0; h < 2; h++) *reinterpret_cast<float4 *>(&s_acc[warp][h * 128 + lane * 4]) = acc[h];
    __syncthreads();
    if (warp == 0) {
        float4 v[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = h * 128 + lane * 4;
            float4 t = *reinterpret_cast<const float4 *>(&s_acc[0][e]);
#pragma unroll
            for (int w = 1; w < 8; w++) {
                const float4 u = *reinterpret_cast<const float4 *>(&s_acc[w][e]);
                t.x += u.x, t.y += u.y, t.z += u.z, t.w += u.w;
            }
            const float l = s_l[e / head_dim];
            v[h] = make_float4(t.x / l, t.y / l, t.z / l, t.w / l);
        }
        if (Q8) {
            quantize_block256(v, lane, (size_t)row, k, chunk, qs, d, sums, sums16);
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) *reinterpret_cast<float4 *>(dst + (size_t)row * k + chunk * 256 + h * 128 + lane * 4) = v[h];
        }
    }
}

// The same merge for at most NT key tiles: a warp for 256 outputs.  All its loads are on their way at once, nothing is shared and no warp waits for
// another, where the kernel above makes two round trips and two barriers for a tile or two a warp.  The sums keep its order: tiles w, w + 8 into
// partial sum w, the eight of them in turn.  (113 rows of 32 heads, 4 tiles: 1808 CTAs of 8 warps 9.1 us, 452 of 4 warps 3.2; a token of 32 heads at 1000: the step 2250 us, 2190.)
constexpr int kMergeWarps = 4;
template <bool Q8, int HEADS, int NT>
__global__ void __launch_bounds__(kMergeWarps * 32) attn_combine_few_kernel(const float *part_o, const float *part_ml, int n_head, int n_splits, int n_blocks,
                                                                            float *__restrict__ dst, int8_t *__restrict__ qs, float *__restrict__ d,
                                                                            int32_t *__restrict__ sums, int32_t *__restrict__ sums16) {
    constexpr int HD = 256 / HEADS;
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31, wg = blockIdx.x * kMergeWarps + (threadIdx.x >> 5), k = n_head * HD, cpr = k / 256;
    if (wg >= n_blocks) return;
    const int row = wg / cpr, chunk = wg % cpr, head0 = chunk * HEADS;
    const size_t first = (size_t)row * n_head + head0;
    float2 ml[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; h++)
        ml[h] = lane < n_splits ? reinterpret_cast<const float2 *>(part_ml)[(first + h) * n_splits + lane] : make_float2(-INFINITY, 0.f);
    float4 p[2][NT];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int e = h * 128 + lane * 4;
        const float *po = part_o + (first + e / HD) * n_splits * HD + e % HD;
#pragma unroll
        for (int s = 0; s < NT; s++)
            if (s < n_splits) p[h][s] = *reinterpret_cast<const float4 *>(po + (size_t)s * HD);
    }
    float wgt[HEADS], l[HEADS];
    int n[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; h++) {
        const float m = warp_max(ml[h].x);
        const bool has = ml[h].y != 0.f;  // not past the row's causal end (a tile with keys has l >= 1, or NaN)
        wgt[h] = has ? expf(ml[h].x - m) : 0.f;
        l[h] = warp_sum(has ? fmaf(wgt[h], ml[h].y, 0.f) : 0.f);
        n[h] = __reduce_max_sync(0xffffffffu, has ? lane + 1 : 0);
    }
    float4 v[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int hh = (h * 128 + lane * 4) / HD;
        float lh = l[0];
        int nh = n[0];
#pragma unroll
        for (int j = 1; j < HEADS; j++)
            if (hh == j) lh = l[j], nh = n[j];
        float4 acc[8];
#pragma unroll
        for (int s = 0; s < NT; s++) {
            float w = 0.f;
#pragma unroll
            for (int j = 0; j < HEADS; j++) {
                const float wj = __shfl_sync(0xffffffffu, wgt[j], s);
                if (hh == j) w = wj;
            }
            float4 &t = acc[s & 7];
            if (s < 8) t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < nh) {  // (nobody writes the sums of the tiles past the causal end)
                const float4 u = p[h][s];
                t.x = fmaf(w, u.x, t.x), t.y = fmaf(w, u.y, t.y), t.z = fmaf(w, u.z, t.z), t.w = fmaf(w, u.w, t.w);
            }
        }
        float4 t = acc[0];
#pragma unroll
        for (int w = 1; w < 8; w++) t.x += acc[w].x, t.y += acc[w].y, t.z += acc[w].z, t.w += acc[w].w;
        v[h] = make_float4(t.x / lh, t.y / lh, t.z / lh, t.w / lh);
    }
    if (Q8) {
        quantize_block256(v, lane, (size_t)row, k, chunk, qs, d, sums, sums16);
    } else {
#pragma unroll
        for (int h = 0; h < 2; h++) *reinterpret_cast<float4 *>(dst + (size_t)row * k + chunk * 256 + h * 128 + lane * 4) = v[h];
    }
}

inline unsigned grid_for(size_t n, int block, const DeviceInfo &dev) {
    const size_t want = (n + (size_t)block - 1) / (size_t)block;
    const size_t cap = (size_t)dev.sm_count * 8;
    return (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
}

}  // namespace

cudaError_t launch_rms_norm(const float *a, const float *b, float *sum_dst, const float *w, float *dst, int rows, int dim, float eps,
                            cudaStream_t st) {
    if (rows <= 0 || dim <= 0) return cudaErrorInvalidValue;
    if (dim % 256 == 0) {  // the block-per-warp kernel, storing f32
        int t = dim / 256 * 32;
        t = t > 1024 ? 1024 : t;
        int8_t *nq = nullptr;
        float *nd = nullptr;
        int32_t *ns = nullptr;
        if (b) return launch_pdl(rms_norm_q8_kernel<true, false>, dim3(rows), dim3(t), 0, st, a, b, sum_dst, w, dim, eps, dst, nq, nd, ns, ns);
        return launch_pdl(rms_norm_q8_kernel<false, false>, dim3(rows), dim3(t), 0, st, a, (const float *)nullptr, nd, w, dim, eps, dst, nq, nd, ns, ns);
    }
    int threads = ((dim / 4 + 31) / 32) * 32;
    threads = threads < 32 ? 32 : (threads > 1024 ? 1024 : threads);
    if (b) return launch_pdl(rms_norm_kernel<true>, dim3(rows), dim3(threads), 0, st, a, b, sum_dst, w, dst, dim, eps);
    return launch_pdl(rms_norm_kernel<false>, dim3(rows), dim3(threads), 0, st, a, (const float *)nullptr, (float *)nullptr, w, dst, dim, eps);
}

cudaError_t launch_rope(const float *x, const int32_t *positions, float *dst, int rows, int n_head, int head_dim, int rope_dim, float theta,
                        int neox, const DeviceInfo &dev, cudaStream_t st) {
    if (rows <= 0 || n_head <= 0 || head_dim <= 0 || rope_dim <= 0 || rope_dim > head_dim || (rope_dim & 1)) return cudaErrorInvalidValue;
    const size_t total = (size_t)rows * n_head * (rope_dim / 2 + head_dim - rope_dim);
    return launch_pdl(rope_kernel, dim3(grid_for(total, 256, dev)), dim3(256), 0, st, x, positions, dst, rows, n_head, head_dim, rope_dim, theta,
                      neox);
}

cudaError_t launch_rope_write_kv(float *q, const float *k, const float *v, const int32_t *positions, void *k_cache, void *v_cache, int rows,
                                 int n_head, int n_kv, int head_dim, float theta, int neox, int rows_per_seq, size_t seq_stride,
                                 const DeviceInfo &dev, cudaStream_t st, int write_pos, const int32_t *block_table, int table_stride, int n_pages) {
    if (rows <= 0 || n_head <= 0 || n_kv <= 0 || head_dim <= 0 || (head_dim & 1) || rows_per_seq <= 0) return cudaErrorInvalidValue;
    const size_t total = (size_t)rows * (n_head + 2 * n_kv) * (head_dim / 2);
    return launch_pdl(rope_write_kv_kernel, dim3(grid_for(total, 256, dev)), dim3(256), 0, st, q, k, v, positions, (__half *)k_cache,
                      (__half *)v_cache, rows, n_head, n_kv, head_dim, theta, neox, rows_per_seq, seq_stride, write_pos, block_table, table_stride,
                      n_pages);
}

cudaError_t launch_write_kv_f16(const float *src, void *cache_at_pos, size_t n, const DeviceInfo &dev, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    return launch_pdl(write_kv_kernel, dim3(grid_for(n, 256, dev)), dim3(256), 0, st, src, (__half *)cache_at_pos, n);
}

size_t attention_workspace_bytes(int q_rows, int n_head, int head_dim, int max_keys) {
    const size_t n_splits = ((size_t)max_keys + kAttnTile - 1) / kAttnTile;
    return (size_t)q_rows * n_head * n_splits * ((size_t)head_dim + 2) * sizeof(float);
}

typedef CUresult (*EncodeAttnFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeAttnFn attn_encode() {
    static EncodeAttnFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeAttnFn>(p);
    }();
    return fn;
}
// Maps of the caches of n_seq sequences, `seq_stride` halves apart, with `n_rows` rows of `row` halves each
static bool attn_maps(const void *k, const void *v, size_t n_rows, int n_seq, size_t row, size_t seq_stride, AttnMaps *maps) {
    EncodeAttnFn enc = attn_encode();
    if (!enc) return false;
    const cuuint64_t dim[3] = {(cuuint64_t)row, (cuuint64_t)n_rows, (cuuint64_t)n_seq}, stride[2] = {(cuuint64_t)row * 2, (cuuint64_t)(n_seq > 1 ? seq_stride : n_rows * row) * 2};
    const cuuint32_t one[3] = {1, 1, 1};
    auto make = [&](CUtensorMap *map, const void *base, int box_rows) {
        const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    return make(&maps->map[0], k, kAttnTile) && make(&maps->map[1], v, kAttnTile) && make(&maps->map[2], k, kBoxRows) && make(&maps->map[3], v, kBoxRows);
}

template <int HD, int G>
static cudaError_t launch_attn_one(dim3 grid, cudaStream_t st, const float *q, const __half *kc, const __half *vc, float *po, float *pml, int rows,
                                   int n_head, int n_kv, int pos, float scale, int n_splits, size_t seq_stride, uint32_t *status, bool boxed,
                                   const int32_t *seq_pos, const int32_t *block_table, int table_stride, int n_pages, const AttnMaps &maps) {
    // the tile needs more than the default 48 KB of dynamic shared memory; the attribute is per device, so it is set
    // on every launch (cheap, allocates nothing) rather than remembered per process
    auto go = [&](auto kernel, int bytes, const auto &m) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        return launch_pdl(kernel, grid, dim3(kAttnThreads), (size_t)bytes, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, seq_pos,
                          block_table, table_stride, n_pages, m);
    };
    return boxed ? go(attn_split_kernel<HD, G, true>, kTileBytes<BoxedTile<HD>>, maps) : go(attn_split_kernel<HD, G, false>, kTileBytes<PaddedTile<HD>>, NoMaps{});
}

template <int HD>
static cudaError_t launch_attn_hd(int group, dim3 grid, cudaStream_t st, const float *q, const __half *kc, const __half *vc, float *po, float *pml,
                                  int rows, int n_head, int n_kv, int pos, float scale, int n_splits, size_t seq_stride, uint32_t *status, bool boxed,
                                  const int32_t *seq_pos, const int32_t *block_table, int table_stride, int n_pages, const AttnMaps &maps) {
    switch (group) {
        case 1: return launch_attn_one<HD, 1>(grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table,
                                                  table_stride, n_pages, maps);
        case 2: return launch_attn_one<HD, 2>(grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table,
                                                  table_stride, n_pages, maps);
        case 4: return launch_attn_one<HD, 4>(grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table,
                                                  table_stride, n_pages, maps);
        case 8: return launch_attn_one<HD, 8>(grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table,
                                                  table_stride, n_pages, maps);
        default: return cudaErrorInvalidValue;
    }
}

template <int G>
static cudaError_t launch_attn_chunk(cudaStream_t st, const float *q, const __half *kc, const __half *vc, float *po, float *pml, int n_seq, int rows,
                                     int n_head, int n_kv, int pos, float scale, int n_splits, size_t seq_stride, uint32_t *status, bool boxed,
                                     const int32_t *seq_pos, const int32_t *block_table, int table_stride, int n_pages, const AttnMaps &maps) {
    constexpr int R = kAttnChunkPairs / G, more = 4 * kAttnChunkPairs * (128 + kAttnPad) * 2 + kAttnChunkPairs * kAttnTile * 4;
    auto go = [&](auto kernel, int bytes, const auto &m) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
        return launch_pdl(kernel, dim3(n_splits, n_kv, n_seq * ((rows + R - 1) / R)), dim3(kAttnThreads), (size_t)bytes, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale,
                          n_splits, seq_stride, status, seq_pos, block_table, table_stride, n_pages, m);
    };
    return boxed ? go(attn_chunk_kernel<G, true>, kTileBytes<BoxedTile<128>> + more, maps) : go(attn_chunk_kernel<G, false>, kTileBytes<PaddedTile<128>> + more, NoMaps{});
}

cudaError_t launch_attention(const float *q, const void *k_cache, const void *v_cache, float *dst, void *workspace, int n_seq, int rows, int n_head,
                             int n_kv, int head_dim, float scale, int pos, size_t seq_stride, int sm_count, cudaStream_t st, uint32_t *status, int8_t *qs, float *d,
                             int32_t *sums, int32_t *sums16, const int32_t *seq_pos, const int32_t *block_table, int table_stride, int n_pages) {
    if (n_seq <= 0 || rows <= 0 || n_head <= 0 || n_kv <= 0 || n_head % n_kv || pos < 0) return cudaErrorInvalidValue;
    const int max_keys = pos + rows, n_splits = (max_keys + kAttnTile - 1) / kAttnTile, q_rows = n_seq * rows;
    if (n_kv > 65535 || q_rows > 65535) return cudaErrorInvalidValue;
    // the tiles are fetched in 16-byte pieces
    if (((uintptr_t)k_cache | (uintptr_t)v_cache) % 16 || seq_stride % 8 || ((size_t)n_kv * head_dim) % 8) return cudaErrorInvalidValue;
    if (block_table && (n_pages < 1 || table_stride < n_splits)) return cudaErrorInvalidValue;
    float *po = static_cast<float *>(workspace);
    float *pml = po + (size_t)q_rows * n_head * n_splits * head_dim;
    const dim3 grid(n_splits, n_kv, q_rows);
    const __half *kc = static_cast<const __half *>(k_cache), *vc = static_cast<const __half *>(v_cache);
    cudaError_t e;
    const int g = n_head / n_kv;
    // Rows of a prompt chunk share a tile where a tile per row takes more than about a wave of CTAs (three fit an SM; two of the shared form, which
    // take 1 us longer) and the shared tile has more than two rows, is nearly full or leaves a single wave.  live: the tiles with keys, each
    // row for itself.  Measured, a tile per row / shared (us, attention and merge), 240 shapes; the rule takes the slower side in none by more than 1 us:
    // 32 heads / 8: 113 rows at 384 40 / 28, 33 at 100 9 / 11 (live 304), 2 at 4000 12.8 / 11.6, 8 at 1500 14.0 / 11.1;  8 / 8: 33 at 0 8.1 / 9.3,
    // 64 at 384 24 / 10;  32 / 32: 64 at 0 23 / 10, 2 at 1500 13.3 / 15.5 (384 shared CTAs);  2 rows of 16 sequences at 1500: 8 / 8 37 / 42, 32 / 4 28 / 24.
    const int rpt = kAttnChunkPairs / (g < 1 ? 1 : g), row_blocks = rpt ? (rows + rpt - 1) / rpt : 0;  // rows of a tile
    const size_t sms = (size_t)(sm_count > 0 ? sm_count : 148);
    auto tiles_to = [](size_t n) { return n / kAttnTile * (n / kAttnTile + 1) / 2 * kAttnTile + n % kAttnTile * (n / kAttnTile + 1); };  // of rows with 1..n keys
    const size_t live = (tiles_to(max_keys) - tiles_to(pos)) * n_kv * n_seq, shared = (size_t)n_splits * n_kv * n_seq * row_blocks;
    const bool chunk = head_dim == 128 && rows > 1 && (g == 1 || g == 2 || g == 4 || g == 8) && 2 * live > 5 * sms &&
                       (rows > 2 * row_blocks || 8 * rows >= 7 * rpt * row_blocks || shared <= 2 * sms);
    // Tensor copies where a tile for each row makes more than two waves of CTAs (three fit an SM), shared tiles more than one (two fit).  Before that the latency of the first byte
    // counts, which is 0.5 to 1 us longer with them: shared tiles, bulk copies of rows / tensor copies, us a call: 32 heads / 8, 64 rows at 128 (256 tiles) 12.1 / 13.1;
    // 8 / 8, 20 rows at 640 (96) 16.0 / 17.2, 300 at 0 (264) 18.3 / 19.2, 64 at 1500 (400) 18.2 / 16.3, 128 at 3000 45 / 42; 32 / 8, 113 at 384 (928) 29.4 / 27.4,
    // 128 at 3000 153 / 142.
    const size_t kv_row = (size_t)n_kv * head_dim;
    AttnMaps maps;
    const bool boxed = (chunk ? live / rows * row_blocks > 2 * sms : (size_t)n_splits * n_kv * q_rows > 6 * sms) && (head_dim == 128 || head_dim == 64) &&
                       attn_maps(k_cache, v_cache, block_table ? (size_t)n_pages * kAttnTile : (size_t)max_keys, block_table ? 1 : n_seq, kv_row, seq_stride, &maps);
#define INFR_CHUNK(G_) launch_attn_chunk<G_>(st, q, kc, vc, po, pml, n_seq, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table, table_stride, n_pages, maps)
    if (chunk)
        e = g == 1 ? INFR_CHUNK(1) : g == 2 ? INFR_CHUNK(2) : g == 4 ? INFR_CHUNK(4) : INFR_CHUNK(8);
    else if (head_dim == 128)
        e = launch_attn_hd<128>(g, grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table, table_stride,
                                n_pages, maps);
    else if (head_dim == 64)
        e = launch_attn_hd<64>(g, grid, st, q, kc, vc, po, pml, rows, n_head, n_kv, pos, scale, n_splits, seq_stride, status, boxed, seq_pos, block_table, table_stride,
                               n_pages, maps);
    else
        return cudaErrorInvalidValue;
#undef INFR_CHUNK
    if (e != cudaSuccess) return e;
    const unsigned merge_ctas = (unsigned)(q_rows * (n_head * head_dim / 256));
    const bool few = merge_ctas <= 2 * sms;
    if (qs && ((n_head * head_dim) % 256 || n_splits > kCombineMaxSplits)) return cudaErrorInvalidValue;  // merged rows straight to int8: whole 256-element blocks
    if (qs || ((n_head * head_dim) % 256 == 0 && n_splits <= kCombineMaxSplits)) {
        if (n_splits <= 16) {
            auto go = [&](auto kernel) {
                return launch_pdl(kernel, dim3((merge_ctas + kMergeWarps - 1) / kMergeWarps), dim3(kMergeWarps * 32), 0, st, (const float *)po, (const float *)pml, n_head,
                                  n_splits, (int)merge_ctas, qs ? nullptr : dst, qs, d, sums, sums16);
            };
            if (head_dim == 128)
                return n_splits <= 8 ? go(qs ? attn_combine_few_kernel<true, 2, 8> : attn_combine_few_kernel<false, 2, 8>)
                                     : go(qs ? attn_combine_few_kernel<true, 2, 16> : attn_combine_few_kernel<false, 2, 16>);
            return n_splits <= 8 ? go(qs ? attn_combine_few_kernel<true, 4, 8> : attn_combine_few_kernel<false, 4, 8>)
                                 : go(qs ? attn_combine_few_kernel<true, 4, 16> : attn_combine_few_kernel<false, 4, 16>);
        }
        auto kernel = qs ? (few ? attn_combine_wide_kernel<true, true> : attn_combine_wide_kernel<true, false>)
                         : (few ? attn_combine_wide_kernel<false, true> : attn_combine_wide_kernel<false, false>);
        return launch_pdl(kernel, dim3(merge_ctas), dim3(256), 0, st, (const float *)po, (const float *)pml, n_head, head_dim, n_splits, qs ? nullptr : dst, qs, d, sums, sums16);
    }
    return launch_pdl(attn_combine_kernel, dim3(q_rows * n_head), dim3(head_dim), 0, st, (const float *)po, (const float *)pml, dst, head_dim, n_splits);
}

cudaError_t launch_rms_norm_q8_pull(const float *a, float *sum_dst, const float *w, int rows, int dim, float eps, int8_t *qs, float *d,
                                    int32_t *sums, int32_t *sums16, const PullArgs &pull, cudaStream_t st) {
    if (rows <= 0 || dim <= 0 || dim % 256 || pull.world < 1 || pull.world > kPushMaxWorld) return cudaErrorInvalidValue;
    int threads = dim / 256 * 32;
    threads = threads > 1024 ? 1024 : threads;
    return launch_pdl(rms_norm_q8_pull_kernel, dim3(rows), dim3(threads), 0, st, a, sum_dst, w, dim, eps, qs, d, sums, sums16, pull);
}

cudaError_t launch_rms_norm_q8(const float *a, const float *b, float *sum_dst, const float *w, int rows, int dim, float eps, int8_t *qs, float *d,
                               int32_t *sums, int32_t *sums16, cudaStream_t st) {
    if (rows <= 0 || dim <= 0 || dim % 256) return cudaErrorInvalidValue;
    int threads = dim / 256 * 32;
    threads = threads > 1024 ? 1024 : threads;
    float *none = nullptr;
    if (b) return launch_pdl(rms_norm_q8_kernel<true, true>, dim3(rows), dim3(threads), 0, st, a, b, sum_dst, w, dim, eps, none, qs, d, sums, sums16);
    return launch_pdl(rms_norm_q8_kernel<false, true>, dim3(rows), dim3(threads), 0, st, a, (const float *)nullptr, none, w, dim, eps, none, qs, d, sums,
                      sums16);
}

cudaError_t launch_gated_silu_q8(const float *gate, const float *up, int rows, int nff, int8_t *qs, float *d, int32_t *sums, int32_t *sums16,
                                 cudaStream_t st) {
    if (rows <= 0 || nff <= 0 || nff % 256) return cudaErrorInvalidValue;
    const long long warps = (long long)rows * (nff / 256);
    return launch_pdl(gated_silu_q8_kernel, dim3((unsigned)((warps * 32 + 255) / 256)), dim3(256), 0, st, gate, up, rows, nff, qs, d, sums, sums16);
}

cudaError_t launch_gated_silu(const float *gate, const float *up, float *dst, size_t n, const DeviceInfo &dev, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    return launch_pdl(gated_silu_kernel, dim3(grid_for(n, 256, dev)), dim3(256), 0, st, gate, up, dst, n);
}

cudaError_t launch_add(const float *a, const float *b, float *dst, size_t n, const DeviceInfo &dev, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    return launch_pdl(add_kernel, dim3(grid_for(n, 256, dev)), dim3(256), 0, st, a, b, dst, n);
}

size_t argmax_workspace_bytes(uint32_t n, uint32_t rows) {
    const uint32_t chunk = 4096, n_chunks = (n + chunk - 1) / chunk;
    return (size_t)rows * n_chunks * 8;
}

cudaError_t launch_argmax(const float *x, uint32_t *dst, void *workspace, uint32_t n, uint32_t rows, cudaStream_t st) {
    if (n == 0 || rows == 0 || rows > 65535) return cudaErrorInvalidValue;
    const uint32_t chunk = 4096, n_chunks = (n + chunk - 1) / chunk;
    float *cv = static_cast<float *>(workspace);
    uint32_t *ci = reinterpret_cast<uint32_t *>(cv + (size_t)rows * n_chunks);
    cudaError_t e = launch_pdl(argmax_stage1_kernel, dim3(n_chunks, rows), dim3(256), 0, st, x, cv, ci, n, chunk);
    if (e != cudaSuccess) return e;
    return launch_pdl(argmax_stage2_kernel, dim3(rows), dim3(256), 0, st, (const float *)cv, (const uint32_t *)ci, dst, n_chunks);
}

}  // namespace infr
