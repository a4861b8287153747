// Mixture-of-experts routing and glue kernels around the grouped expert GEMMs.
//
// Follows the staged Op::MoeFfn of crates/infr-cpu/src/lib.rs:2264-2984 for the qwen3moe family
// (split gate/up banks, softmax gating, top-k by stable descending sort, optional renormalisation,
// SiLU gate, output-side weighting):
//   router logits  : F32 router rows against the raw f32 activations with the reference's `dot`
//                    (8 FMA lanes, lanes summed in order, kernels.rs:6557-6573) -> same bits as the CPU
//   route          : softmax over all experts with max shift, sequential sums (lib.rs:2427-2436),
//                    top-k = repeated arg-max with the lower expert id winning ties (:2527-2529),
//                    w = p / max(sum p_sel, 1e-20) * scale (:2536-2538)
//   bucket         : pairs (row, rank) grouped by expert, in (row, rank) order inside an expert
//                    (:2554-2587), plus the 8-row work items of the grouped GEMM
//   swiglu_quant   : act = silu(g) * u per pair (kernels.rs:6578-6597), re-quantised per 256
//                    (lib.rs:2862-2873) with the arithmetic of quantize.cu
//   combine        : out[r] += w * y in rank order, multiply and add rounded separately (:2970-2982)
#include "kernels.h"
#include "pdl.cuh"
#include "q8_code.cuh"

namespace infr {

// logits[r, e] = dot(router[e, :], x[r, :]).  Eight lanes per dot product replay the eight accumulators of the CPU
// `dot` (lane j takes elements j, 8 + j, ... in order, the lanes are then summed in order; rows are whole groups of eight).  A lane has 4 rows x 4 experts, a warp 4 x 16, a block of four warps 16 x 16.  Columns come 512 at a time, a bulk copy a row (the copy engine
// takes a row in 45 cycles, however short), into a ring of three; the row pitch (520 words) puts the four groups of a warp on disjoint banks.
// What bounds it: shared memory delivers 128 bytes a cycle to registers however many lanes share an address, so that the work per value read counts: 8
// reads feed 16 multiply-adds (128 experts x 2048, 256 rows: 4 warps x 256 x 8 = 8192 cycles a block), where 6 fed 8.  Behind that one warp a scheduler.
// Measured there: 13.6 us (the first copies land after 3.3, 16000 cycles are reads and multiply-adds), 18.7 before; 512 rows of 4096: 46, 66.  (Columns
// 256 at a time 18.7; a row and two experts a thread by 16-byte reads and packed multiply-adds 21.7.)
constexpr int kRtRows = 16, kRtExperts = 16, kRtK = 512, kRtPitch = kRtK + 8, kRtBuf = (kRtRows + kRtExperts) * kRtPitch, kRtRing = 3;
__global__ void __launch_bounds__(128) moe_router_kernel(const float *__restrict__ router, const float *x,
                                                         float *__restrict__ logits, int rows, int ne, int n_expert, uint32_t *__restrict__ status) {
    extern __shared__ __align__(16) float s_rt[];  // [kRtRing][16 rows, 16 router rows][kRtPitch]
    __shared__ uint64_t bars[kRtRing];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 3, j = lane & 7;
    const int r0 = blockIdx.x * kRtRows, e0 = blockIdx.y * kRtExperts;
    const int rl = warp * 4;  // the warp's first row; its group has experts grp, grp + 4, ...
    const int n_chunks = (ne + kRtK - 1) / kRtK;
    auto su32 = [](const void *p) { return (uint32_t)__cvta_generic_to_shared(p); };
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRtRing; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&bars[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_go();
    pdl_wait();
    // columns c * kRtK .. of the block's rows and router rows (rows past the last are not read: what is there goes into sums that are not stored)
    auto source = [&](int i) { return i < kRtRows ? (r0 + i < rows ? x + (size_t)(r0 + i) * ne : nullptr) : (e0 + i - kRtRows < n_expert ? router + (size_t)(e0 + i - kRtRows) * ne : nullptr); };
    auto fetch = [&](int c) {  // (warp 0: a row a lane)
        const float *src = source(lane);
        const uint32_t bytes = (uint32_t)min(kRtK, ne - c * kRtK) * 4, bar = su32(&bars[c % kRtRing]), n = __popc(__ballot_sync(0xffffffffu, src != nullptr));
        if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n * bytes) : "memory");
        __syncwarp();
        if (src)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             su32(s_rt + (c % kRtRing) * kRtBuf + lane * kRtPitch)),
                         "l"(src + c * kRtK), "r"(bytes), "r"(bar)
                         : "memory");
    };
    auto landed = [&](int c) {
        for (uint32_t i = 0; i < (1u << 22); i++) {
            uint32_t ok;
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok)
                         : "r"(su32(&bars[c % kRtRing])), "r"((uint32_t)(c / kRtRing) & 1u)
                         : "memory");
            if (ok) return true;
        }
        return false;
    };
    if (warp == 0)
        for (int c = 0; c < kRtRing && c < n_chunks; c++) fetch(c);
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 16; a++) (&acc[0][0])[a] = 0.f;
    for (int c0 = 0; c0 < n_chunks; c0++) {
        const int kc = min(kRtK, ne - c0 * kRtK);
        const float *buf = s_rt + (c0 % kRtRing) * kRtBuf;
        if (!__syncthreads_and(landed(c0))) {  // give up; the copies in flight get their own limit (chunk 1 is the first whose landing asks for another)
            if (threadIdx.x == 0) atomicExch(status, 14u);
            for (int c = c0 + 1; c < kRtRing + (c0 > 1 ? c0 - 1 : 0) && c < n_chunks; c++) landed(c);
            return;
        }
        if (warp == 0 && c0 >= 1 && c0 - 1 + kRtRing < n_chunks) {  // everybody has finished with the columns before these
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            fetch(c0 - 1 + kRtRing);
        }
        const float *xa = buf + rl * kRtPitch + j, *wa = buf + (kRtRows + grp) * kRtPitch + j;
#pragma unroll 8
        for (int c = 0; c < kc; c += 8) {
            float v[4], w[4];
#pragma unroll
            for (int a = 0; a < 4; a++) v[a] = xa[a * kRtPitch + c], w[a] = wa[4 * a * kRtPitch + c];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) acc[a][b] = fmaf(w[b], v[a], acc[a][b]);
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) {
            // s = ((((acc0 + acc1) + acc2) + ...) + acc7)
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < 8; k++) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, acc[a][b], grp * 8 + k));
            const int r = r0 + rl + a, e = e0 + grp + 4 * b;
            if (j == ((a * 4 + b) & 7) && r < rows && e < n_expert) logits[(size_t)r * n_expert + e] = sum;
        }
}

// One warp per row.  n_expert <= 1024.
__global__ void __launch_bounds__(128) moe_route_kernel(const float *logits, int rows, int n_expert, int n_used,
                                                        float scale, int norm_w, int32_t *__restrict__ sel_ids,
                                                        float *__restrict__ sel_w) {
    pdl_go();
    pdl_wait();
    extern __shared__ float s_p[];  // [warps][n_expert]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = blockIdx.x * (blockDim.x >> 5) + warp;
    if (r >= rows) return;
    float *p = s_p + (size_t)warp * n_expert;
    const float *lg = logits + (size_t)r * n_expert;
    float mx = -INFINITY;
    for (int e = lane; e < n_expert; e += 32) mx = fmaxf(mx, lg[e]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    for (int e = lane; e < n_expert; e += 32) p[e] = expf(lg[e] - mx);
    __syncwarp();
    float psum = 0.f;
    if (lane == 0)
        for (int e = 0; e < n_expert; e++) psum = __fadd_rn(psum, p[e]);  // the CPU sums in index order
    psum = __shfl_sync(0xffffffffu, psum, 0);
    for (int e = lane; e < n_expert; e += 32) p[e] = __fdiv_rn(p[e], psum);
    __syncwarp();
    // top-k: k rounds of arg-max; ties go to the lower expert id (what a stable descending sort does)
    float wsum = 0.f;
    float myw = 0.f;  // lane k keeps the k-th selected probability (n_used <= 32)
    int myid = 0;
    for (int k = 0; k < n_used; k++) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int e = lane; e < n_expert; e += 32) {
            const float v = p[e];
            if (v > best) {
                best = v;
                bi = e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (bi == 0x7fffffff) {
            // No probability compared greater than -inf: the row is all NaN (a NaN or infinite logit poisons the
            // softmax sum).  The CPU's stable sort leaves such a row in index order, so take the lowest expert
            // not selected yet; its NaN weight travels on as it does there.
            for (int e = lane; e < n_expert; e += 32)
                if (p[e] != -INFINITY) {
                    bi = e;
                    break;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) bi = min(bi, __shfl_xor_sync(0xffffffffu, bi, o));
            if (bi < n_expert) best = p[bi];
        }
        wsum = __fadd_rn(wsum, best);
        if (lane == k) {
            myw = best;
            myid = bi < n_expert ? bi : 0;
        }
        if (lane == 0 && bi < n_expert) p[bi] = -INFINITY;  // never compares greater than the running best again
        __syncwarp();
    }
    wsum = fmaxf(wsum, 1e-20f);
    if (lane < n_used) {
        sel_ids[(size_t)r * n_used + lane] = myid;
        sel_w[(size_t)r * n_used + lane] = norm_w ? __fmul_rn(__fdiv_rn(myw, wsum), scale) : __fmul_rn(myw, scale);
    }
}

// One CTA of 32 warps lists the routed pairs by expert, in (row, rank) order inside an expert, and cuts every
// expert's pairs into work items of up to `item_rows` rows (8 for the grouped GEMV, 64 = one token tile for the
// grouped tensor-memory GEMM).
//   pair_row[p], pair_of_slot[r * n_used + rank] = p, item_{expert,p0,cnt}[], n_items
// Expert parallelism: only experts [e_lo, e_lo + n_local) are listed (item_expert is the index inside this
// rank's banks); pairs routed elsewhere get pair_of_slot = -1 and contribute nothing to this rank's output.
__global__ void __launch_bounds__(1024) moe_bucket_kernel(const int32_t *sel_ids, int rows, int n_used, int n_expert,
                                                          int e_lo, int n_local, int item_rows,
                                                          int32_t *__restrict__ pair_row, int32_t *__restrict__ pair_of_slot,
                                                          int32_t *__restrict__ item_expert, int32_t *__restrict__ item_p0,
                                                          int32_t *__restrict__ item_cnt, int32_t *__restrict__ n_items,
                                                          int32_t *__restrict__ counts_out, int n_chunks) {
    pdl_go();
    pdl_wait();
    // A stable counting sort over chunks of 32 pairs: hist[chunk][expert] = pairs of the expert inside the chunk
    // (lanes with the same expert find each other with a match), an exclusive scan down the chunks gives the place of
    // a chunk's first such pair inside its expert, and a pair's place is that plus its rank among the lanes before it:
    // (row, rank) order is kept and the work is linear in the number of pairs.
    __shared__ int s_cnt[1024], s_off[1024], s_ioff[1024];
    __shared__ int2 s_wsum[32];
    extern __shared__ int32_t s_hist[];  // [n_chunks][n_expert]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_pairs = rows * n_used;
    for (int i = threadIdx.x; i < n_chunks * n_expert; i += 1024) s_hist[i] = 0;
    __syncthreads();
    // the expert of pair i as this rank sees it: -1 for another rank's expert or an id outside the bank
    auto local_expert = [&](int i) {
        if (i >= n_pairs) return -1;
        const int e = sel_ids[i];
        return (e < e_lo || e >= e_lo + n_local || e < 0 || e >= n_expert) ? -1 : e;
    };
    for (int c = warp; c < n_chunks; c += 32) {
        const int e = local_expert(c * 32 + lane);
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && (same & ((1u << lane) - 1u)) == 0) s_hist[c * n_expert + e] = __popc(same);
    }
    __syncthreads();
    // (n_expert <= 1024: an expert a thread)
    int run = 0;
    if ((int)threadIdx.x < n_expert) {
        int32_t *h = s_hist + threadIdx.x;
        int c = 0;
        for (; c + 8 <= n_chunks; c += 8) {  // eight reads in flight
            int t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = h[(c + k) * n_expert];
#pragma unroll
            for (int k = 0; k < 8; k++) h[(c + k) * n_expert] = run, run += t[k];
        }
        for (; c < n_chunks; c++) {
            const int t = h[c * n_expert];
            h[c * n_expert] = run;
            run += t;
        }
        s_cnt[threadIdx.x] = run;
        if (counts_out) counts_out[threadIdx.x] = run;
    }
    // exclusive sums over the experts of their pairs and their items: inside the warps, then over the warps
    const int its = (run + item_rows - 1) / item_rows;
    int off = run, ioff = its;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, off, o), b = __shfl_up_sync(0xffffffffu, ioff, o);
        if (lane >= o) off += a, ioff += b;
    }
    if (lane == 31) s_wsum[warp] = make_int2(off, ioff);
    __syncthreads();
    if (warp == 0) {
        int2 v = s_wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, v.x, o), b = __shfl_up_sync(0xffffffffu, v.y, o);
            if (lane >= o) v.x += a, v.y += b;
        }
        s_wsum[lane] = v;
        if (lane == 31) *n_items = v.y;
    }
    __syncthreads();
    if ((int)threadIdx.x < n_expert) {
        const int2 before = warp ? s_wsum[warp - 1] : make_int2(0, 0);
        s_off[threadIdx.x] = before.x + off - run;
        s_ioff[threadIdx.x] = before.y + ioff - its;
    }
    __syncthreads();
    for (int c = warp; c < n_chunks; c += 32) {
        const int i = c * 32 + lane;
        const int e = local_expert(i);
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        if (i < n_pairs) {
            int q = -1;  // pairs routed to an expert that is not listed contribute nothing to this rank's output
            if (e >= 0) {
                q = s_off[e] + s_hist[c * n_expert + e] + __popc(same & ((1u << lane) - 1u));
                pair_row[q] = i / n_used;
            }
            pair_of_slot[i] = q;
        }
    }
    for (int e = warp; e < n_expert; e += 32) {
        const int cnt = s_cnt[e];
        for (int c = lane * item_rows; c < cnt; c += 32 * item_rows) {
            const int it = s_ioff[e] + c / item_rows;
            item_expert[it] = e - e_lo;
            item_p0[it] = s_off[e] + c;
            item_cnt[it] = cnt - c < item_rows ? cnt - c : item_rows;
        }
    }
}

// One warp per (pair, 256-block): act = silu(gate) * up, then quantize_q8 of that block.
__global__ void __launch_bounds__(256) moe_swiglu_quant_kernel(const float *gate, const float *up,
                                                               int n_pairs, int nff, int8_t *__restrict__ qs, float *__restrict__ d,
                                                               int32_t *__restrict__ sums, int32_t *__restrict__ sums16,
                                                               float *__restrict__ act_out) {
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int nbk = nff / 256;
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wg >= (long long)n_pairs * nbk) return;
    const int p = (int)(wg / nbk), b = (int)(wg % nbk);
    const size_t base = (size_t)p * nff + (size_t)b * 256 + lane * 8;
    float v[8];
    float am = 0.f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float4 g4 = *reinterpret_cast<const float4 *>(gate + base + h * 4);
        const float4 u4 = *reinterpret_cast<const float4 *>(up + base + h * 4);
        const float gg[4] = {g4.x, g4.y, g4.z, g4.w}, uu[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float sg = __fdiv_rn(gg[i], __fadd_rn(1.0f, expf(-gg[i])));
            v[h * 4 + i] = __fmul_rn(sg, uu[i]);
            am = fmaxf(am, fabsf(v[h * 4 + i]));
        }
    }
    if (act_out) {
#pragma unroll
        for (int i = 0; i < 8; i++) act_out[base + i] = v[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float dd = am / 127.0f;
    const float id = dd > 0.0f ? 1.0f / dd : 0.0f;
    const uint2 pk = make_uint2(q8_codes4(make_float4(v[0], v[1], v[2], v[3]), id), q8_codes4(make_float4(v[4], v[5], v[6], v[7]), id));
    int sum = q8_sum4(pk.x) + q8_sum4(pk.y);
    *reinterpret_cast<uint2 *>(qs + base) = pk;
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (sums16 && (lane & 1) == 0) sums16[((size_t)p * nbk + b) * 16 + (lane >> 1)] = sum;  // Q6_K banks: sums per 16 codes
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if ((lane & 3) == 0) sums[((size_t)p * nbk + b) * 8 + (lane >> 2)] = sum;
    if (lane == 0) d[(size_t)p * nbk + b] = dd;
}

// out[r, i] = sum over ranks (in rank order) of w[r, rank] * y[pair_of_slot[r, rank], i].
__global__ void __launch_bounds__(256) moe_combine_kernel(const float *y_pairs, const int32_t *pair_of_slot,
                                                          const float *sel_w, int rows, int n_used, int ne,
                                                          float *__restrict__ out) {
    pdl_go();
    pdl_wait();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * ne) return;
    const int r = (int)(idx / ne), i = (int)(idx % ne);
    float o = 0.f;
    for (int k = 0; k < n_used; k++) {
        const int p = pair_of_slot ? pair_of_slot[(size_t)r * n_used + k] : r * n_used + k;
        if (p < 0) continue;  // routed to an expert of another rank
        o = __fadd_rn(o, __fmul_rn(sel_w[(size_t)r * n_used + k], y_pairs[(size_t)p * ne + i]));
    }
    out[idx] = o;
}

cudaError_t launch_moe_router(const float *router, const float *x, float *logits, int rows, int ne, int n_expert,
                              const DeviceInfo &dev, uint32_t *status, cudaStream_t st) {
    if (rows < 1 || n_expert < 1) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)((rows + kRtRows - 1) / kRtRows), (unsigned)((n_expert + kRtExperts - 1) / kRtExperts));
    if (grid.y > 65535 || ne % 8 || (((uintptr_t)x | (uintptr_t)router) & 15)) return cudaErrorInvalidValue;
    // A few rows: a warp an expert and four rows, all columns staged at once, as long as its CTAs are four waves at most.  Measured, tiles /
    // rows (us a layer; waves): 27 rows, 128 experts x 2048 15 / 7.4 (the router alone); 64 rows, 64 experts x 2048 (0.6) 85 / 71,
    // 128 x 4096 (3.5) 155 / 145, 512 x 1024 (2.3) 72 / 77, 256 x 4096 (6.9) 163 / 175; 48 rows, 192 x 6144 (3.9) 205 / 195, 256 x 6144
    // (5.2) 208 / 213; 32 rows, 512 x 2048 (2.3) 86 / 87, 512 x 4096 (6.9) 127 / 144.
    const size_t row_smem = moe_router_row_smem(ne);
    const size_t row_ctas = (size_t)((n_expert + 3) / 4) * ((rows + 3) / 4), fit = (size_t)dev.max_smem_optin / (row_smem + 1024);
    if (rows <= 64 && row_ctas <= 4 * (size_t)dev.sm_count * (fit < 16 ? fit : 16)) {
        const cudaError_t e = launch_moe_router_row(router, x, logits, rows, ne, n_expert, st);
        if (e != cudaErrorInvalidValue) return e;
        cudaGetLastError();
    }
    const size_t smem = (size_t)kRtRing * kRtBuf * 4;
    cudaError_t e = cudaFuncSetAttribute(moe_router_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(moe_router_kernel, grid, dim3(128), smem, st, router, x, logits, rows, ne, n_expert, status);
}

cudaError_t launch_moe_route(const float *logits, int rows, int n_expert, int n_used, float scale, int norm_w,
                             int32_t *sel_ids, float *sel_w, cudaStream_t st) {
    if (n_expert > 1024 || n_used > 32 || n_used > n_expert) return cudaErrorInvalidValue;
    if (n_expert <= 256) return launch_moe_route_rows(logits, rows, n_expert, n_used, scale, norm_w, sel_ids, sel_w, st);
    const int warps = 4;
    return launch_pdl(moe_route_kernel, dim3((unsigned)((rows + warps - 1) / warps)), dim3(warps * 32), (size_t)warps * n_expert * 4, st, logits, rows,
                      n_expert, n_used, scale, norm_w, sel_ids, sel_w);
}

cudaError_t launch_moe_bucket(const int32_t *sel_ids, int rows, int n_used, int n_expert, int e_lo, int n_local, int item_rows,
                              int32_t *pair_row, int32_t *pair_of_slot, int32_t *item_expert, int32_t *item_p0, int32_t *item_cnt,
                              int32_t *n_items, int32_t *counts_out, cudaStream_t st) {
    if (n_expert > 1024 || item_rows < 1) return cudaErrorInvalidValue;
    const int n_chunks = (rows * n_used + 31) / 32;
    const size_t hist_bytes = (size_t)n_chunks * n_expert * 4;
    if (hist_bytes > 200 * 1024) return cudaErrorInvalidValue;  // ~51 000 pairs of 128 experts; more would need a multi-CTA sort
    cudaError_t e = cudaFuncSetAttribute(moe_bucket_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_bytes);
    if (e != cudaSuccess) return e;
    return launch_pdl(moe_bucket_kernel, dim3(1), dim3(1024), hist_bytes, st, sel_ids, rows, n_used, n_expert, e_lo, n_local, item_rows, pair_row,
                      pair_of_slot, item_expert, item_p0, item_cnt, n_items, counts_out, n_chunks);
}

cudaError_t launch_moe_swiglu_quant(const float *gate, const float *up, int n_pairs, int nff, int8_t *qs, float *d,
                                    int32_t *sums, int32_t *sums16, float *act_out, cudaStream_t st) {
    if (nff % 256) return cudaErrorInvalidValue;
    const long long warps = (long long)n_pairs * (nff / 256);
    return launch_pdl(moe_swiglu_quant_kernel, dim3((unsigned)((warps * 32 + 255) / 256)), dim3(256), 0, st, gate, up, n_pairs, nff, qs, d, sums, sums16,
                      act_out);
}

cudaError_t launch_moe_combine(const float *y_pairs, const int32_t *pair_of_slot, const float *sel_w, int rows, int n_used,
                               int ne, float *out, cudaStream_t st) {
    const long long n = (long long)rows * ne;
    return launch_pdl(moe_combine_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, y_pairs, pair_of_slot, sel_w, rows, n_used, ne, out);
}

}  // namespace infr
