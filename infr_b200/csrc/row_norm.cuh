// RMSNorm of one row by one CTA (optionally of a + b, written to sum_dst); dim % 256 == 0.  Shared by the kernels that store the scaled row
// as f32, as int8 codes and as the tensor-memory GEMM's operand, which therefore agree bit for bit.
#pragma once
#include <cuda_runtime.h>

#include "pdl.cuh"

namespace infr {

// Sum of squares of four values with every product and sum rounded on its own (no fused multiply-add): two kernels
// that share this get the same bits whatever the compiler does around it, and it is how the CPU forms the sum.
__device__ __forceinline__ float sumsq4(const float4 v) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y)), __fmul_rn(v.z, v.z)), __fmul_rn(v.w, v.w));
}

__device__ __forceinline__ float row_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Warp c owns the 256-element blocks c, c + warps, ...; with one block per warp (dim <= 256 * warps, the launcher's
// choice up to dim 8192) the row stays in registers between the sum of squares and the scaling.
// out(block, v): lane l holds elements 4l..4l+3 (v[0]) and 128+4l.. (v[1]) of the scaled block.  s_part: 32 floats of shared memory.
template <bool ADD, class Out>
__device__ __forceinline__ void rms_norm_row(const float *a, const float *b, float *sum_dst, const float *__restrict__ w, int dim, float eps, size_t row, float *s_part,
                                             const Out &out) {
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
    const size_t base = row * dim;
    float4 x[2];
    float ss = 0.f;
    for (int chunk = warp; chunk < chunks; chunk += nw) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = chunk * 256 + h * 128 + lane * 4;
            float4 v = *reinterpret_cast<const float4 *>(a + base + e);
            if (ADD) {
                const float4 u = *reinterpret_cast<const float4 *>(b + base + e);
                v.x += u.x, v.y += u.y, v.z += u.z, v.w += u.w;
                *reinterpret_cast<float4 *>(sum_dst + base + e) = v;
            }
            ss = __fadd_rn(ss, sumsq4(v));
            x[h] = v;
        }
    }
    ss = row_warp_sum(ss);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    const float s = 1.0f / sqrtf(row_warp_sum(lane < nw ? s_part[lane] : 0.f) / (float)dim + eps);  // (every warp for itself: no second barrier)
    const float *src = (ADD ? sum_dst : a) + base;  // re-read by the warp that wrote it
    for (int chunk = warp; chunk < chunks; chunk += nw) {
        float4 v[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = chunk * 256 + h * 128 + lane * 4;
            if (!in_regs) {
                x[h] = *reinterpret_cast<const float4 *>(src + e);
                g[h] = *reinterpret_cast<const float4 *>(w + e);
            }
            v[h] = make_float4(x[h].x * s * g[h].x, x[h].y * s * g[h].y, x[h].z * s * g[h].z, x[h].w * s * g[h].w);
        }
        out(chunk, v);
    }
}

__device__ __forceinline__ float silu_mul(float g, float u) { return g / (1.0f + expf(-g)) * u; }

}  // namespace infr
