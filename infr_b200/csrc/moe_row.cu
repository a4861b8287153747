// One decoded token of an MoE layer (one row, f32 activations: crates/infr-cpu/src/lib.rs:2359 keeps a single row off the int8 path)
// in three launches:
//   router     logits, bit for bit the CPU's `dot` (kernels.rs:6557-6573: eight FMA lanes, summed in order)
//   gate / up  every CTA routes the row for itself (moe_route_row, the arithmetic of moe_route_kernel), then a warp per (expert, FFN
//              row) multiplies the gate and the up row and stores silu(g) * u (kernels.rs:6578-6597)
//   down       a warp per output row multiplies it with every selected expert and adds the results in rank order, multiply and add
//              rounded separately (:2970-2982)
// Weights are dequantised with the two roundings of crates/infr-gguf/src/dequant.rs:31-47 (scale * code, + minimum), products are
// f32 fused multiply-adds, as in gemv.cu's f32 kernels; the two weights of a byte make a packed f32 pair.
//
// What bounds it: the chain of launches and round trips to memory (9.3 MB of weights are 1.4 us), the routing in front of the gate
// weights (a serial sum over the experts, k rounds of arg-max) and issue slots: four packed operations and two byte permutes a pair of
// weights.  Measured (hidden 2048, 128 experts, top-8, 768 wide): seven launches of the general path 61 us (three GEMVs of 11.6 us,
// whose lanes read activations 64 bytes apart: 16-way bank conflicts; a router on 8 CTAs 11.6 us), these three 24 us: router 4, gate
// and up 11, down 7.
//
// Only the weights are const __restrict__ (pdl.cuh): the ids were, and the down kernel's load of them went above its wait.  Wherever the
// gate / up launch left SMs idle, so that the next one was resident beside it, it took whatever the scratch held.
#include "f32x2.cuh"
#include "kernels.h"
#include "pdl.cuh"

#include <cuda_fp16.h>

namespace infr {
namespace {

constexpr int kRowThreads = 512, kRowWarps = kRowThreads / 32;

__device__ __forceinline__ float both(u64 v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ float hf(uint32_t bits) { return __half2float(__ushort_as_half((unsigned short)(bits & 0xffffu))); }

// ---- router: warp = expert, its groups of eight lanes a row each.  The rows go to shared memory in one round trip; eight lanes replay
// the CPU's accumulators.  (Row pitch ne + 8: the four groups on disjoint banks.)
constexpr int kRtWarps = 4, kRtRowsCta = 4;
__global__ void __launch_bounds__(kRtWarps * 32) moe_router_row_kernel(const float *__restrict__ router, const float *x, float *__restrict__ logits,
                                                                       int rows, int ne, int n_expert) {
    extern __shared__ __align__(16) float s_rt[];  // [the experts' rows][rows][ne + 8]
    pdl_go();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pitch = ne + 8, e = blockIdx.x * kRtWarps + warp, r0 = blockIdx.y * kRtRowsCta;
    if (e < n_expert) {
        const float4 *w = reinterpret_cast<const float4 *>(router + (size_t)e * ne);
        float4 *sw = reinterpret_cast<float4 *>(s_rt + (size_t)warp * pitch);
#pragma unroll 8
        for (int i = lane; i < ne / 4; i += 32) sw[i] = __ldg(w + i);
    }
    if (r0 + warp < rows) {  // (one row a warp)
        const float4 *p = reinterpret_cast<const float4 *>(x + (size_t)(r0 + warp) * ne);
        float4 *sx = reinterpret_cast<float4 *>(s_rt + (size_t)(kRtWarps + warp) * pitch);
#pragma unroll 8
        for (int i = lane; i < ne / 4; i += 32) sx[i] = p[i];
    }
    __syncthreads();
    const int grp = lane >> 3, j = lane & 7, r = min(r0 + grp, rows - 1);  // (groups past the last row repeat it)
    if (e >= n_expert) return;
    const float *w = s_rt + (size_t)warp * pitch + j, *xr = s_rt + (size_t)(kRtWarps + r - r0) * pitch + j;
    float acc = 0.f;
#pragma unroll 16
    for (int c = 0; c < ne; c += 8) acc = fmaf(w[c], xr[c], acc);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, acc, grp * 8 + k));
    if (j == 0 && r0 + grp < rows) logits[(size_t)r * n_expert + e] = sum;
}
static_assert(kRtRowsCta == kRtWarps, "a warp stages one expert row and one activation row");

// ---- routing of one row by one warp: moe_route_kernel's operations in the same order.  EPL: experts of a lane (e = lane + 32 i),
// in registers.  p: [32 EPL] floats of shared memory, for the sum in index order.
template <int EPL>
__device__ __forceinline__ void moe_route_row(const float *logits, float *p, int n_expert, int n_used, float scale, int norm_w, int lane, int &id,
                                              float &weight) {
    float v[EPL], mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < EPL; i++) v[i] = lane + 32 * i < n_expert ? logits[lane + 32 * i] : -INFINITY;
#pragma unroll
    for (int i = 0; i < EPL; i++) mx = fmaxf(mx, v[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int i = 0; i < EPL; i++)
        if (lane + 32 * i < n_expert) p[lane + 32 * i] = v[i] = expf(v[i] - mx);
    __syncwarp();
    float psum = 0.f;
    int e = 0;
#pragma unroll 4
    for (; e + 4 <= n_expert; e += 4) {  // the CPU sums in index order
        const float4 q = *reinterpret_cast<const float4 *>(p + e);
        psum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(psum, q.x), q.y), q.z), q.w);
    }
    for (; e < n_expert; e++) psum = __fadd_rn(psum, p[e]);
    // Keys order like the probabilities (none is negative); 0: taken, NaN or no expert.
    uint32_t key[EPL];
#pragma unroll
    for (int i = 0; i < EPL; i++) {
        v[i] = __fdiv_rn(v[i], psum);
        key[i] = lane + 32 * i < n_expert && v[i] >= 0.f ? __float_as_uint(v[i]) + 1u : 0u;
    }
    uint32_t taken = 0;  // of the lane's experts
    float wsum = 0.f, myw = 0.f;
    int myid = 0;
    for (int k = 0; k < n_used; k++) {
        uint32_t best = 0u;
#pragma unroll
        for (int i = 0; i < EPL; i++) best = max(best, key[i]);
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        // the lowest expert with that key; with none left but NaN, the lowest that is not taken
        uint32_t mine = 0x7fffffffu;
#pragma unroll
        for (int i = EPL - 1; i >= 0; i--)
            if (top ? key[i] == top : (lane + 32 * i < n_expert && !(taken >> i & 1))) mine = lane + 32 * i;
        const int bi = (int)__reduce_min_sync(0xffffffffu, mine);
        float value = __uint_as_float(top - 1u);
        if (!top) {
            float nan = 0.f;
#pragma unroll
            for (int i = 0; i < EPL; i++)
                if (i == bi >> 5) nan = v[i];
            value = __shfl_sync(0xffffffffu, nan, bi & 31);
        }
        wsum = __fadd_rn(wsum, value);
        if (lane == k) myw = value, myid = bi;
        if (lane == (bi & 31)) {
            taken |= 1u << (bi >> 5);
#pragma unroll
            for (int i = 0; i < EPL; i++)
                if (i == bi >> 5) key[i] = 0u;
        }
    }
    wsum = fmaxf(wsum, 1e-20f);
    id = myid;
    weight = norm_w ? __fmul_rn(__fdiv_rn(myw, wsum), scale) : __fmul_rn(myw, scale);
}

// ---- routing of many rows: one warp each.  (128 experts, 8 of them, 256 rows: 4.2 us; probabilities in shared memory and shuffles for every round
// of the choice, as moe_route_kernel has them for more than 256 experts, 6.4.)
constexpr int kRouteWarps = 4;
template <int EPL>
__global__ void __launch_bounds__(kRouteWarps * 32) moe_route_rows_kernel(const float *logits, int rows, int n_expert, int n_used, float scale, int norm_w,
                                                                          int32_t *__restrict__ sel_ids, float *__restrict__ sel_w) {
    __shared__ __align__(16) float s_p[kRouteWarps][32 * EPL];
    pdl_go();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * kRouteWarps + warp;
    if (r >= rows) return;
    int id;
    float w;
    moe_route_row<EPL>(logits + (size_t)r * n_expert, s_p[warp], n_expert, n_used, scale, norm_w, lane, id, w);
    if (lane < n_used) sel_ids[(size_t)r * n_used + lane] = id, sel_w[(size_t)r * n_used + lane] = w;
}

// Activations of a 256-element block as the lanes consume them: four lanes, lane t the sub-blocks 2t and 2t + 1; 16-byte unit
// u * 4 + t holds elements 2u, 2u + 1 of both: (lo, hi, lo, hi).  Blocks are 64 bytes more than their kilobyte apart: the two blocks of
// eight lanes' 16-byte reads lie on different banks.
constexpr int kBlockPitch = 68;  // float4
__device__ __forceinline__ void stage_block_pairs(const float *x, float4 *s, int n, int tid, int nthr) {
    for (int i = tid; i < n / 4; i += nthr) {
        const int b = i >> 6, r = i & 63, u = r >> 2, t = r & 3;
        const float *src = x + b * 256 + t * 64 + 2 * u;
        const float2 lo = *reinterpret_cast<const float2 *>(src), hi = *reinterpret_cast<const float2 *>(src + 32);
        s[b * kBlockPitch + r] = make_float4(lo.x, hi.x, lo.y, hi.y);
    }
}
// The lane's 64 weights of a block: header, its 32 bytes.
struct Piece {
    uint4 h, q0, q1;
};
__device__ __forceinline__ Piece fetch_piece(const uint8_t *blk, int t) {
    const uint4 *p = reinterpret_cast<const uint4 *>(blk);
    return Piece{__ldg(p), __ldg(p + 1 + 2 * t), __ldg(p + 2 + 2 * t)};
}
// Against its activations, for N matrices.  A pair = the low and the high nibble of a byte.
template <int N>
__device__ __forceinline__ void block_dot(const Piece (&w)[N], const float4 *s_x, int t, u64 (&acc)[N]) {
    u64 sc[N], mn[N];
#pragma unroll
    for (int m = 0; m < N; m++) {
        // get_scale_min_k4 (crates/infr-gguf/src/dequant.rs:73-83) of sub-blocks 2t, 2t + 1
        const uint4 h = w[m].h;
        uint32_t s = t < 2 ? h.y & 0x3F3F3F3Fu : (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
        uint32_t n = t < 2 ? h.z & 0x3F3F3F3Fu : ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
        const int sh = 16 * (t & 1);
        s >>= sh, n >>= sh;
        const float d = hf(h.x), dm = hf(h.x >> 16);
        sc[m] = f2_pack(__fmul_rn(d, (float)(s & 0xFFu)), __fmul_rn(d, (float)((s >> 8) & 0xFFu)));
        mn[m] = f2_pack(__fmul_rn(dm, (float)(-(int)(n & 0xFFu))), __fmul_rn(dm, (float)(-(int)((n >> 8) & 0xFFu))));
    }
    const u64 neg = f2_pack(-8388608.0f, -8388608.0f);
    // a byte under the exponent of 2^23 is 2^23 + byte
    auto under = [](uint32_t v, int k) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u + k)); };
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint32_t lo[N], hi[N];
#pragma unroll
        for (int m = 0; m < N; m++) {
            const uint4 q = i < 4 ? w[m].q0 : w[m].q1;
            const uint32_t v = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
            lo[m] = v & 0x0F0F0F0Fu, hi[m] = (v >> 4) & 0x0F0F0F0Fu;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const ulonglong2 xv = *reinterpret_cast<const ulonglong2 *>(s_x + (2 * i + h) * 4 + t);
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int m = 0; m < N; m++)
                    acc[m] = f2_fma(f2_add(f2_mul(sc[m], f2_add(f2_pack(under(lo[m], 2 * h + k), under(hi[m], 2 * h + k)), neg)), mn[m]), k ? xv.y : xv.x, acc[m]);
        }
    }
}

// Gate and up of every selected expert, SiLU.  Task = (rank, FFN row); a warp's four-lane group g takes blocks g, g + 8, ...
constexpr int kEpl = 4;  // up to 128 experts
__global__ void __launch_bounds__(kRowThreads, 1) moe_gate_up_row_kernel(const float *logits, const float *x, const uint8_t *__restrict__ gate,
                                                                        const uint8_t *__restrict__ up, float *__restrict__ act, int32_t *__restrict__ sel_ids,
                                                                        float *__restrict__ sel_w, int ne, int nff, int n_expert, int n_used, float scale, int norm_w) {
    extern __shared__ __align__(16) float4 s_x[];  // [ne / 256][kBlockPitch]
    __shared__ __align__(16) float s_p[32 * kEpl];
    __shared__ int s_id[32];
    pdl_go();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (warp == 0) {
        int id;
        float w;
        moe_route_row<kEpl>(logits, s_p, n_expert, n_used, scale, norm_w, lane, id, w);
        if (lane < n_used) {
            s_id[lane] = id;
            if (blockIdx.x == 0) sel_ids[lane] = id, sel_w[lane] = w;
        }
    } else {
        stage_block_pairs(x, s_x, ne, threadIdx.x - 32, kRowThreads - 32);
    }
    __syncthreads();
    const int nb = ne >> 8, tasks = n_used * nff, stride = gridDim.x * kRowWarps;
    const uint32_t row_bytes = (uint32_t)nb * 144u;
    Piece w[2];
    auto fetch = [&](int task, int b) {
        const int r = task / nff;
        const size_t off = ((size_t)s_id[r] * nff + (size_t)(task - r * nff)) * row_bytes + (size_t)b * 144;
        if (b < nb) w[0] = fetch_piece(gate + off, t), w[1] = fetch_piece(up + off, t);
    };
    int task = blockIdx.x * kRowWarps + warp;
    if (task < tasks) fetch(task, g);
    for (; task < tasks; task += stride) {
        u64 acc[2] = {0ull, 0ull};
        for (int b = g; b - g < nb; b += 8) {
            const Piece cur[2] = {w[0], w[1]};
            // what comes next is in flight while this is multiplied
            if (b - g + 8 < nb)
                fetch(task, b + 8);
            else if (task + stride < tasks)
                fetch(task + stride, g);
            if (b < nb) block_dot<2>(cur, s_x + b * kBlockPitch, t, acc);
        }
        float vg = both(acc[0]), vu = both(acc[1]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            vg += __shfl_xor_sync(0xffffffffu, vg, o);
            vu += __shfl_xor_sync(0xffffffffu, vu, o);
        }
        if (lane == 0) act[task] = __fmul_rn(__fdiv_rn(vg, __fadd_rn(1.0f, expf(-vg))), vu);
    }
}

// Down of every selected expert and the weighted sum in rank order.  Warp = output row; its eight groups of four lanes take 8 / P ranks
// at a time, P groups a rank's blocks.  (CTAs of 256 threads and 64 registers find room beside the launch before, but spill: 31 us a layer
// for 24.)
__global__ void __launch_bounds__(kRowThreads, 1) moe_down_row_kernel(const uint8_t *__restrict__ down, const float *act, const int32_t *sel_ids,
                                                                      const float *sel_w, float *__restrict__ dst, int ne, int nff, int n_used, int P) {
    extern __shared__ __align__(16) float4 s_x[];  // [n_used][nff / 256][kBlockPitch]
    __shared__ int s_id[32];
    __shared__ float s_w[32];
    pdl_go();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if ((int)threadIdx.x < n_used) s_id[threadIdx.x] = sel_ids[threadIdx.x], s_w[threadIdx.x] = sel_w[threadIdx.x];
    const int nb = nff >> 8, R = 8 / P, gr = g / P, gb = g % P;
    const int per = (nb + P - 1) / P, steps = (n_used + R - 1) / R * per;  // step u: rank (u / per) R + gr, block (u % per) P + gb
    const uint32_t row_bytes = (uint32_t)nb * 144u;
    __syncthreads();
    constexpr int kPre = 4;  // steps in flight
    int row = blockIdx.x * kRowWarps + warp;  // (every warp has one: ne is a multiple of 256, and a CTA has 16 of them)
    Piece w[kPre];
    int fr, fb;  // the next step to fetch: its rank and block
    auto fetch = [&](Piece &p) {
        if (fr < n_used && fb < nb) p = fetch_piece(down + ((size_t)s_id[fr] * ne + row) * row_bytes + (size_t)fb * 144, t);
        fb += P;
        if (fb - gb >= per * P) fb = gb, fr += R;
    };
    auto fetch_first = [&]() {
        fr = gr, fb = gb;
#pragma unroll
        for (int k = 0; k < kPre; k++) fetch(w[k]);
    };
    fetch_first();
    stage_block_pairs(act, s_x, n_used * nff, threadIdx.x, kRowThreads);  // the first weights are on their way
    __syncthreads();
    while (true) {
        float o = 0.f;
        u64 acc[1] = {0ull};
        int rank0 = 0, i = 0;
        for (int u0 = 0; u0 < steps; u0 += kPre) {
#pragma unroll
            for (int k = 0; k < kPre; k++) {
                if (u0 + k < steps) {
                    const int rank = rank0 + gr, b = i * P + gb;
                    if (rank < n_used && b < nb) {
                        const Piece cur[1] = {w[k]};
                        block_dot<1>(cur, s_x + (rank * nb + b) * kBlockPitch, t, acc);
                    }
                    fetch(w[k]);
                    if (++i == per) {
                        // R ranks are done: their sums, added in rank order by every lane alike
                        float v = both(acc[0]);
                        for (int sft = 2 * P; sft > 0; sft >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sft);
                        for (int r = 0; r < R; r++) {
                            const float y = __shfl_sync(0xffffffffu, v, r * 4 * P);
                            if (rank0 + r < n_used) o = __fadd_rn(o, __fmul_rn(s_w[rank0 + r], y));
                        }
                        acc[0] = 0ull, i = 0, rank0 += R;
                    }
                }
            }
        }
        if (lane == 0) dst[row] = o;
        row += gridDim.x * kRowWarps;
        if (row >= ne) break;
        fetch_first();
    }
}

size_t pairs_smem(size_t n) { return n / 256 * kBlockPitch * 16; }

}  // namespace

// One row, Q4_K banks; false: the general path (more than 128 experts, activations that do not fit shared memory, unaligned operands).
bool moe_row_takes(int ne, int nff, int n_expert, int n_used, const float *x, const float *router, const uint8_t *gate, const uint8_t *up, const uint8_t *down) {
    if (ne % 256 || nff % 256 || n_used > 32 || n_expert > 32 * kEpl) return false;
    if (pairs_smem(ne) > 200 * 1024 || pairs_smem((size_t)n_used * nff) > 200 * 1024) return false;
    return (((uintptr_t)x | (uintptr_t)router | (uintptr_t)gate | (uintptr_t)up | (uintptr_t)down) & 15) == 0;
}

// A few rows (launch_moe_router draws the line), columns in whole groups of eight; cudaErrorInvalidValue: the tiles take it.
size_t moe_router_row_smem(int ne) { return (size_t)(kRtRowsCta + kRtWarps) * (ne + 8) * 4; }
cudaError_t launch_moe_router_row(const float *router, const float *x, float *logits, int rows, int ne, int n_expert, cudaStream_t st) {
    const size_t smem = moe_router_row_smem(ne);
    if (rows < 1 || ne % 8 || smem > 220 * 1024 || (((uintptr_t)router | (uintptr_t)x) & 15)) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(moe_router_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((n_expert + kRtWarps - 1) / kRtWarps), (unsigned)((rows + kRtRowsCta - 1) / kRtRowsCta));
    return launch_pdl(moe_router_row_kernel, grid, dim3(kRtWarps * 32), smem, st, router, x, logits, rows, ne, n_expert);
}
// cudaErrorInvalidValue: more experts than a warp's registers take here.
cudaError_t launch_moe_route_rows(const float *logits, int rows, int n_expert, int n_used, float scale, int norm_w, int32_t *sel_ids, float *sel_w, cudaStream_t st) {
    if (n_expert > 256) return cudaErrorInvalidValue;
    auto kernel = n_expert <= 32 ? moe_route_rows_kernel<1> : n_expert <= 64 ? moe_route_rows_kernel<2> : n_expert <= 128 ? moe_route_rows_kernel<4> : moe_route_rows_kernel<8>;
    return launch_pdl(kernel, dim3((unsigned)((rows + kRouteWarps - 1) / kRouteWarps)), dim3(kRouteWarps * 32), 0, st, logits, rows, n_expert, n_used, scale, norm_w,
                      sel_ids, sel_w);
}
cudaError_t launch_moe_gate_up_row(const float *logits, const float *x, const uint8_t *gate, const uint8_t *up, float *act, int32_t *sel_ids, float *sel_w, int ne,
                                   int nff, int n_expert, int n_used, float scale, int norm_w, const DeviceInfo &dev, cudaStream_t st) {
    const size_t smem = pairs_smem(ne);
    cudaError_t e = cudaFuncSetAttribute(moe_gate_up_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int grid = (n_used * nff + kRowWarps - 1) / kRowWarps;
    grid = grid < dev.sm_count ? grid : dev.sm_count;
    return launch_pdl(moe_gate_up_row_kernel, dim3((unsigned)grid), dim3(kRowThreads), smem, st, logits, x, gate, up, act, sel_ids, sel_w, ne, nff, n_expert,
                      n_used, scale, norm_w);
}
cudaError_t launch_moe_down_row(const uint8_t *down, const float *act, const int32_t *sel_ids, const float *sel_w, float *dst, int ne, int nff, int n_used,
                                const DeviceInfo &dev, cudaStream_t st) {
    const size_t smem = pairs_smem((size_t)n_used * nff);
    cudaError_t e = cudaFuncSetAttribute(moe_down_row_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    // groups of a rank: the fewest steps, of those the fewest groups
    const int nb = nff / 256;
    int P = 1, best = 1 << 30;
    for (int p = 1; p <= 8; p *= 2) {
        const int steps = (n_used + 8 / p - 1) / (8 / p) * ((nb + p - 1) / p);
        if (steps < best) best = steps, P = p;
    }
    int grid = (ne + kRowWarps - 1) / kRowWarps;
    grid = grid < dev.sm_count ? grid : dev.sm_count;
    return launch_pdl(moe_down_row_kernel, dim3((unsigned)grid), dim3(kRowThreads), smem, st, down, act, sel_ids, sel_w, dst, ne, nff, n_used, P);
}

}  // namespace infr
