// Batched GEMM C[m, out_f] = Q8x32(x)[m, in_f] * W^T for Q2_0 weights (64 two-bit codes and one f16 scale in 18 bytes), more than
// 8 rows, any row length, on the warp-level int8 matrix unit (mma.sync m16n8k32).
//
// Arithmetic of vec_dot_q2_0 (crates/infr-cpu/src/kernels.rs:5641-5668): per 64-element block
//     C += d * (d8_0 * s_0 + d8_1 * s_1),   s_h = sum over 32 elements of (code - 1) * q8      (exact int32)
// A block's terms are added to a stage's sum (8 blocks) first and that to the running one, so that hundreds of blocks do not
// round one by one.
//
// Why not tcgen05: an activation group of 32 elements has a scale of its own, so every 32 elements of K each output's sum has to
// come out of the matrix unit and be scaled.  The tensor-memory form of this kernel spent its time on that (a drain and a round of
// barriers per 64 elements).  Here one mma.sync IS one group, its sums are born in the registers of the warp that scales them, and
// the conversion to f32 is part of the instruction: the accumulator starts as the bit pattern of 1.5 * 2^23, so the int32 result
// read as f32 is 1.5 * 2^23 + s, and one packed subtraction gives s exactly.
//
// What bounds it: issue and the f32 pipe.  Per 32 rows x 40 tokens x 64 elements a warp issues
// 315 instructions, of them 20 matrix instructions and 100 packed f32 operations (2.5 per output and group), and moves that put the
// start value into the accumulators (a conversion of the int32 sums instead costs as much); 0.49 instructions a cycle and scheduler, f32
// pipe 41 %, matrix unit 25 % busy.
// Measured (us, whole call, against the tensor-memory form for rows of whole 512-element chunks, the 8-row walk for others):
// 14336 -> 4096, 77 rows 78 -> 41;  4096 -> 14336, 12 rows 32 -> 20, 64 rows 46 -> 38, 512 rows 282 -> 232;  4096 -> 4096, 32 rows
// 21 -> 13;  4160 -> 1000, 40 rows 52 -> 13;  14336 -> 4096, 1024 rows 502 -> 417.
//
// Split: CTA = 256 weight rows x up to 80 tokens x a range of K; 16 warps = 8 groups of 32 rows x 2 halves, which share the tokens
// (more than 40) or the blocks of K (up to 40: the unpacking is not repeated).  Sixteen warps of 128 registers, because two warps to
// a scheduler left it idle 60 % of the cycles (80 tokens x 4096 -> 14336); the running sums of the stages are therefore kept in
// shared memory, each warp its own, the current stage's in registers.
// Weights: rows start on any even address, so the 16-byte-aligned superset of a stage's bytes of a row is fetched, in 16-byte
// cp.async pieces, and read from the remainder (one bulk copy per row and stage instead kept the copy engine busy ~45 cycles per
// row: 28 us of the 46 that 80 tokens x 4096 -> 14336 took); double-buffered, the first ones fetched before the dependency wait.  Activations:
// gemm_q2_prep_kernel lays them out in the order the lanes consume them, so that half a stage is one bulk copy.  Split K writes
// partial results that a second kernel adds in split order.
// Every wait is bounded; a CTA that gives up records a status word, waits (bounded) for its copies and returns.
#include "f32x2.cuh"
#include "gemv_common.cuh"
#include "pdl.cuh"
#include "q8_code.cuh"

namespace infr {
namespace {

constexpr int kRowsCta = 256;   // weight rows of a CTA
constexpr int kThreadsQ2 = 512;
constexpr int kStageBlk = 8;    // 64-element blocks of a weight stage: 144 bytes of a row
constexpr int kHalfBlk = 4;     // of an activation stage
constexpr int kPieces = 10;     // 16-byte pieces that 144 bytes from any even address touch
constexpr int kRowPitch = 176;  // 144 bytes + up to 14 before and after, rounded up; 44 words: eight rows on distinct banks
constexpr int kMaxNtw = 5;       // groups of 8 tokens of a warp
constexpr uint32_t kSpinQ2 = 1u << 22;
constexpr uint32_t kMagic = 0x4B400000u;  // f32 bits of 1.5 * 2^23

__device__ __forceinline__ uint32_t q2_su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool q2_wait(uint32_t bar, uint32_t parity, uint32_t spins) {
    for (uint32_t i = 0; i < spins; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void q2_copy(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// D = A(16x32, s8) * B(32x8, s8) + c (1.5 * 2^23 as f32 bits, four times)
__device__ __forceinline__ void q2_mma(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const uint4 &c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
}
// Activations: per (token tile, 64-element block) a record of NT x 512 bytes of codes, NT x 64 bytes of scales.
//   codes  [n][lane g * 4 + t][group h][2 words]: token 8 n + g, elements 32 h + 8 t + {0, 2, 4, 6} and + {1, 3, 5, 7}
//   scales [n][t][group h][2]: tokens 8 n + 2 t, + 1
constexpr int record_bytes(int nt) { return nt * 576; }

// One warp per (token, 256 elements); lane l owns elements [8l, 8l + 8) = lane t = l % 4 of group l / 4.  Quantises per 32 with
// the operations of quantize.cu in the same order (crates/infr-cpu/src/quant.rs:97-117).  Tokens past the last one are zero.
__global__ void __launch_bounds__(256) gemm_q2_prep_kernel(const float *x, int m, int nt, int in_f, uint8_t *__restrict__ act, int n_tok) {
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31, nc = (in_f + 255) >> 8, nb = in_f >> 6;
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wg >= (long long)n_tok * nc) return;
    const int T = (int)(wg / nc), e0 = (int)(wg % nc) * 256 + lane * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (T < m && e0 < in_f) {
        const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)T * in_f + e0);
        const float4 p = xp[0], q = xp[1];
        v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = p.w, v[4] = q.x, v[5] = q.y, v[6] = q.z, v[7] = q.w;
    }
    float am = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[i]));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    if (e0 >= in_f) return;
    const float d = am / 127.0f;
    const float id = d > 0.0f ? 1.0f / d : 0.0f;
    const int tile = T / (8 * nt), tt = T % (8 * nt), n = tt >> 3, g = tt & 7, b = e0 >> 6, h = (lane >> 2) & 1, t = lane & 3;
    uint8_t *rec = act + ((size_t)tile * nb + b) * record_bytes(nt);
    *reinterpret_cast<uint2 *>(rec + n * 512 + (g * 4 + t) * 16 + h * 8) = make_uint2(q8_codes4(make_float4(v[0], v[2], v[4], v[6]), id), q8_codes4(make_float4(v[1], v[3], v[5], v[7]), id));
    if (t == 0) *reinterpret_cast<float *>(rec + nt * 512 + n * 64 + (g >> 1) * 16 + h * 8 + (g & 1) * 4) = d;
}

struct Q2Mat {
    const uint8_t *w;
    float *c;  // [m, out_f] (K split: the first of kz partial results)
    int out_f, kz;
};

// NTW: groups of 8 tokens of a warp.  KH: the two halves of the warps share the blocks, else the tokens.
template <int NTW, bool KH>
__global__ void __launch_bounds__(kThreadsQ2, 1) gemm_q2_kernel(Q2Mat m1, Q2Mat m2, const uint8_t *act, int m, int nb, int tiles,
                                                                uint32_t *__restrict__ status) {
    constexpr int NT = KH ? NTW : 2 * NTW, kRaw = kRowsCta * kRowPitch, kRec = record_bytes(NT), kAct = kHalfBlk * kRec, kSums = 4 * NTW;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bars[2];  // activations
    __shared__ uint4 s_magic;
    uint8_t *s_act = smem + 2 * kRaw;
    u64 *s_sum = reinterpret_cast<u64 *>(s_act + 2 * kAct);  // [16 warps][4 NTW][32 lanes]: pairs of running sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, rg = warp & 7, hf = warp >> 3;
    pdl_go();
    if (tid == 0) {
        s_magic = make_uint4(kMagic, kMagic, kMagic, kMagic);
#pragma unroll
        for (int i = 0; i < 2; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(q2_su32(&bars[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // work item: the first matrix, then the second; K split fastest, then weight rows (neighbouring CTAs share activations), then tokens
    const int items1 = (m1.out_f + kRowsCta - 1) / kRowsCta * tiles * m1.kz;
    const bool second = (int)blockIdx.x >= items1;
    const uint8_t *W = second ? m2.w : m1.w;
    const int of = second ? m2.out_f : m1.out_f, kz = second ? m2.kz : m1.kz, row_tiles = (of + kRowsCta - 1) / kRowsCta;
    const int i0 = (int)blockIdx.x - (second ? items1 : 0), ks = i0 % kz, r = i0 / kz, tt = r / row_tiles, row0 = r % row_tiles * kRowsCta;
    const int b_begin = (int)((long long)ks * nb / kz), b_end = (int)((long long)(ks + 1) * nb / kz);
    const int n_half = (b_end - b_begin + kHalfBlk - 1) / kHalfBlk;
    const size_t row_bytes = (size_t)nb * 18;

    // the K range's i-th stage of every row, consecutive threads taking consecutive 16-byte pieces of a row
    auto fetch_w = [&](int i) {
        const int b0 = b_begin + i * kStageBlk, n = min(kStageBlk, b_end - b0);
#pragma unroll
        for (int k = 0; k < kRowsCta * kPieces / kThreadsQ2; k++) {
            const int idx = tid + k * kThreadsQ2, row = idx / kPieces, piece = idx - row * kPieces;
            const size_t start = (size_t)W + (size_t)(row0 + row) * row_bytes + (size_t)b0 * 18;
            if (row0 + row < of && piece * 16 < (int)(start & 15) + n * 18)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(q2_su32(smem + (i & 1) * kRaw + row * kRowPitch + piece * 16)),
                             "l"((start & ~(size_t)15) + piece * 16)
                             : "memory");
        }
    };
    auto fetch_a = [&](int i) {
        const int b0 = b_begin + i * kHalfBlk, n = min(kHalfBlk, b_end - b0);
        q2_copy(q2_su32(s_act + (i & 1) * kAct), act + ((size_t)tt * nb + b0) * kRec, (uint32_t)(n * kRec), q2_su32(&bars[i & 1]));
    };
    // (the weights do not depend on the kernels before this one)
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (2 * i < n_half) fetch_w(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    pdl_wait();
    if (tid == 0)
        for (int i = 0; i < 2 && i < n_half; i++) fetch_a(i);

    // The K range of the lane's weight rows g, g + 8, g + 16, g + 24 of the group's 32 starts up to 14 bytes into their slots (a stage is a whole
    // number of 16-byte units).  Rows past the matrix are not fetched: what the slot holds is multiplied and never stored.
    const uint8_t *rp[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int rr = rg * 32 + g + 8 * j;
        rp[j] = smem + rr * kRowPitch + (((size_t)W + (size_t)(row0 + rr) * row_bytes + (size_t)b_begin * 18) & 15);
    }
    u64 *my_sum = s_sum + (size_t)warp * kSums * 32 + lane;
    const uint4 magic = s_magic;  // from memory: as a constant it is moved into place again for every instruction
    const u64 neg = f2_dup(-__uint_as_float(kMagic));
    u64 part[2][NTW][2];  // the stage's sums: [rows 0..15 / 16..31][token group][rows g / g + 8], tokens 2t and 2t + 1
    int dead = 0;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // the first stage has landed for everybody
    for (int i = 0; i < n_half; i++) {
        const int st = i >> 1;
        if (!(i & 1)) {
#pragma unroll
            for (int k = 0; k < kSums; k++) (&part[0][0][0])[k] = 0ull;
        }
        dead = !q2_wait(q2_su32(&bars[i & 1]), (uint32_t)st & 1u, kSpinQ2);
        const int n = min(kHalfBlk, b_end - b_begin - i * kHalfBlk);
        const uint8_t *ab = s_act + (i & 1) * kAct + lane * 16 + (KH ? 0 : hf * NTW * 512);
        const uint8_t *sb = s_act + (i & 1) * kAct + NT * 512 + t * 16 + (KH ? 0 : hf * NTW * 64);
        const int wo = (st & 1) * kRaw + (i & 1) * kHalfBlk * 18;
#pragma unroll 1
        for (int blk = KH ? hf : 0; blk < n; blk += KH ? 2 : 1) {
            uint32_t a[2][2][4];  // [rows 0..15 / 16..31][group][operand word]
            float dw[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned short *p = reinterpret_cast<const unsigned short *>(rp[j] + wo + blk * 18);
                dw[j] = h2f(p[0]);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    // eight codes: even ones to one word, odd ones to the other, each through a table of code - 1
                    const uint32_t u = p[1 + 4 * h + t];
                    a[j >> 1][h][j & 1] = __byte_perm(0x020100FFu, 0, u & 0x3333u);
                    a[j >> 1][h][2 + (j & 1)] = __byte_perm(0x020100FFu, 0, (u >> 2) & 0x3333u);
                }
            }
#pragma unroll
            for (int k = 0; k < NTW; k++) {
                const uint4 bv = *reinterpret_cast<const uint4 *>(ab + blk * kRec + k * 512);
                const ulonglong2 d8 = *reinterpret_cast<const ulonglong2 *>(sb + blk * kRec + k * 64);
#pragma unroll
                for (int mt = 0; mt < 2; mt++) {
                    uint32_t c0[4], c1[4];
                    q2_mma(c0, a[mt][0], bv.x, bv.y, magic);
                    q2_mma(c1, a[mt][1], bv.z, bv.w, magic);
#pragma unroll
                    for (int v = 0; v < 2; v++) {
                        const u64 f0 = f2_add(f2_pack(c0[2 * v], c0[2 * v + 1]), neg), f1 = f2_add(f2_pack(c1[2 * v], c1[2 * v + 1]), neg);
                        part[mt][k][v] = f2_fma(f2_dup(dw[2 * mt + v]), f2_fma(f1, d8.y, f2_mul(f0, d8.x)), part[mt][k][v]);
                    }
                }
            }
        }
        if ((i & 1) || i == n_half - 1) {
#pragma unroll
            for (int k = 0; k < kSums; k++) my_sum[k * 32] = st ? f2_add(my_sum[k * 32], (&part[0][0][0])[k]) : (&part[0][0][0])[k];
        }
        if (i & 1) asm volatile("cp.async.wait_group 0;" ::: "memory");  // the next stage's weights
        // everybody has read the buffers (and nobody gave up): they are filled again
        if (__syncthreads_or(dead)) {
            if (tid == 0) atomicExch(status, 13u);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            for (int k = i; k <= i + 1 && k < n_half; k++) q2_wait(q2_su32(&bars[k & 1]), (uint32_t)(k >> 1) & 1u, 1u << 14);
            return;
        }
        if ((i & 1) && 2 * (st + 2) < n_half) {
            fetch_w(st + 2);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (tid == 0 && i + 2 < n_half) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            fetch_a(i + 2);
        }
    }
    // (the last round's barrier has made all sums visible)
    float *C = (second ? m2.c : m1.c) + (size_t)ks * m * of;
    const int tok0 = tt * 8 * NT + (KH ? 0 : hf * NTW * 8) + 2 * t;
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
        if (KH && mt != hf) continue;  // halves of K: each half of the warps adds and stores one half of the rows
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int row = row0 + rg * 32 + mt * 16 + v * 8 + g;
            if (row >= of) continue;
#pragma unroll
            for (int k = 0; k < NTW; k++) {
                const int idx = ((mt * NTW + k) * 2 + v) * 32;
                u64 s = my_sum[idx];
                if (KH) s = f2_add(s_sum[(size_t)rg * kSums * 32 + lane + idx], s_sum[(size_t)(rg + 8) * kSums * 32 + lane + idx]);
                const int tok = tok0 + 8 * k;
                if (tok < m) C[(size_t)tok * of + row] = __uint_as_float((uint32_t)s);
                if (tok + 1 < m) C[(size_t)(tok + 1) * of + row] = __uint_as_float((uint32_t)(s >> 32));
            }
        }
    }
}

template <int NTW, bool KH>
cudaError_t launch_ntw(int grid, cudaStream_t st, Q2Mat m1, Q2Mat m2, const uint8_t *act, int m, int nb, int tiles, uint32_t *status) {
    constexpr int NT = KH ? NTW : 2 * NTW;
    constexpr size_t smem = (size_t)2 * kRowsCta * kRowPitch + (size_t)2 * kHalfBlk * record_bytes(NT) + (size_t)16 * 4 * NTW * 32 * 8;
    static_assert(smem <= 227 * 1024 - 64, "shared memory");
    cudaError_t e = cudaFuncSetAttribute(gemm_q2_kernel<NTW, KH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(gemm_q2_kernel<NTW, KH>, dim3((unsigned)grid), dim3(kThreadsQ2), smem, st, m1, m2, act, m, nb, tiles, status);
}

// Tokens are cut evenly: the fewest tiles of at most 80, each of the fewest groups of 8 (pairs of groups above 40 tokens).
int q2_tiles(int m) { return (m + 79) / 80; }
int q2_nt(int m) {
    const int tiles = q2_tiles(m), nt = ((m + tiles - 1) / tiles + 7) / 8;
    return nt <= kMaxNtw ? nt : (nt + 1) / 2 * 2;
}
int q2_row_tiles(int out_f1, int out_f2) { return (out_f1 + kRowsCta - 1) / kRowsCta + (out_f2 + kRowsCta - 1) / kRowsCta; }

// How many ways K is split across CTAs (one fits an SM).  Estimate in microseconds, from 12..512 tokens against 2048..28672 rows of
// 1024..14336: a block takes 0.18 + 0.105 NT, a CTA's start and end 2.5; the kernel that adds the parts 2.5, their words, written
// and read through L2, 1.2e-6 each.
int q2_splits(int m, int in_f, int out_f1, int out_f2, const DeviceInfo &dev) {
    const int nb = in_f / 64, items = q2_row_tiles(out_f1, out_f2) * q2_tiles(m);
    const double blk = 0.18 + 0.105 * q2_nt(m);
    int best = 1;
    double best_cost = 1e30;
    for (int kz = 1; kz <= 32 && 4 * kz <= nb; kz++) {
        const int waves = (items * kz + dev.sm_count - 1) / dev.sm_count;
        const double cost = waves * ((double)nb / kz * blk + 2.5) + (kz > 1 ? 2.5 + 1.2e-6 * kz * m * ((double)out_f1 + out_f2) : 0.0);
        if (cost < best_cost * 0.98) best = kz, best_cost = cost;
    }
    return best;
}

// Up to 16 rows a pair has the bits of two calls: each matrix is split as it would be alone.  (12 rows of 4096 -> 2 x 14336: 2 ways each,
// 40 us; 1 way as both heights together would have it, 36; walked 8 rows at a time 68.)  More rows: by both heights together.
constexpr int kPairBits = 16;
void q2_pair_splits(int m, int in_f, int out_f1, int out_f2, const DeviceInfo &dev, int &kz1, int &kz2) {
    kz1 = kz2 = q2_splits(m, in_f, out_f1, out_f2, dev);
    if (out_f2 && m <= kPairBits) kz1 = q2_splits(m, in_f, out_f1, 0, dev), kz2 = q2_splits(m, in_f, out_f2, 0, dev);
}

__device__ __forceinline__ void add_to(float4 &a, const float4 &v) { a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w; }
__device__ __forceinline__ void add_to(float &a, float v) { a += v; }

// y[i] = part[0][i] + part[1][i] + ... in split order (the same bits on every run), for two results (n = 0: none).  V = float4, or float
// where a result's size is not a multiple of four or its address not 16-byte aligned.
template <typename V>
__global__ void __launch_bounds__(256) gemm_q2_sum_kernel(const V *part, V *__restrict__ y, size_t n1, int kz, const V *part2,
                                                          V *__restrict__ y2, size_t n2, int kz2) {
    pdl_go();
    pdl_wait();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n1 + n2) return;
    if (i >= n1) i -= n1, part = part2, y = y2, n1 = n2, kz = kz2;
    V acc = part[i];
    for (int s = 1; s < kz; s++) add_to(acc, part[(size_t)s * n1 + i]);
    y[i] = acc;
}
template <typename V>
cudaError_t launch_sum(const float *p, float *y, size_t n1, int kz, const float *p2, float *y2, size_t n2, int kz2, cudaStream_t st) {
    constexpr size_t L = sizeof(V) / 4;
    return launch_pdl(gemm_q2_sum_kernel<V>, dim3((unsigned)(((n1 + n2) / L + 255) / 256)), dim3(256), 0, st, reinterpret_cast<const V *>(p),
                      reinterpret_cast<V *>(y), n1 / L, kz, reinterpret_cast<const V *>(p2), reinterpret_cast<V *>(y2), n2 / L, kz2);
}

size_t q2_align(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

bool gemm_q2_takes(int in_f) { return in_f > 0 && in_f % 64 == 0; }
// Scratch: the activation records (gemm_q2_record_bytes), then the parts of a split K (gemm_q2_partial_bytes).
size_t gemm_q2_record_bytes(int m, int in_f) { return q2_align((size_t)q2_tiles(m) * (in_f / 64) * record_bytes(q2_nt(m))); }
size_t gemm_q2_partial_bytes(int m, int in_f, int out_f1, int out_f2, const DeviceInfo &dev) {
    int kz1, kz2;
    q2_pair_splits(m, in_f, out_f1, out_f2, dev, kz1, kz2);
    return q2_align(((kz1 > 1 ? (size_t)kz1 * out_f1 : 0) + (kz2 > 1 ? (size_t)kz2 * out_f2 : 0)) * m * 4);
}

cudaError_t launch_gemm_q2_prep(const float *x, void *records, int m, int in_f, cudaStream_t st) {
    if (m < 1 || !gemm_q2_takes(in_f) || (uintptr_t)x % 16) return cudaErrorInvalidValue;
    const int nt = q2_nt(m), n_tok = q2_tiles(m) * 8 * nt;
    const size_t warps = (size_t)n_tok * ((in_f + 255) / 256);
    return launch_pdl(gemm_q2_prep_kernel, dim3((unsigned)((warps + 7) / 8)), dim3(256), 0, st, x, m, nt, in_f, static_cast<uint8_t *>(records), n_tok);
}

cudaError_t launch_gemm_q2(const uint8_t *w, const void *records, float *c, float *partials, int m, int in_f, int out_f, const DeviceInfo &dev,
                           uint32_t *status, cudaStream_t st, const uint8_t *w2, float *c2, int out_f2) {
    if (m <= 8 || out_f < 1 || !gemm_q2_takes(in_f) || (w2 && out_f2 < 1)) return cudaErrorInvalidValue;
    if (!w2) out_f2 = 0;
    int kz1, kz2;
    q2_pair_splits(m, in_f, out_f, out_f2, dev, kz1, kz2);
    // elements whose parts are to be added
    const size_t n1 = kz1 > 1 ? (size_t)m * out_f : 0, n2 = kz2 > 1 ? (size_t)m * out_f2 : 0;
    if (n1 + n2 && !partials) return cudaErrorInvalidValue;
    float *p2 = partials + kz1 * n1;
    const Q2Mat m1{w, n1 ? partials : c, out_f, kz1}, m2{w2, n2 ? p2 : c2, out_f2, kz2};
    const int tiles = q2_tiles(m), grid = (q2_row_tiles(out_f, 0) * kz1 + q2_row_tiles(out_f2, 0) * kz2) * tiles;
    const uint8_t *act = static_cast<const uint8_t *>(records);
    const int nb = in_f / 64;
    cudaError_t e = cudaErrorInvalidValue;
    switch (q2_nt(m)) {
    case 2: e = launch_ntw<2, true>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 3: e = launch_ntw<3, true>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 4: e = launch_ntw<4, true>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 5: e = launch_ntw<5, true>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 6: e = launch_ntw<3, false>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 8: e = launch_ntw<4, false>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    case 10: e = launch_ntw<5, false>(grid, st, m1, m2, act, m, nb, tiles, status); break;
    }
    if (e != cudaSuccess || !(n1 + n2)) return e;
    const bool v4 = n1 % 4 == 0 && n2 % 4 == 0 && (!n1 || (uintptr_t)c % 16 == 0) && (!n2 || (uintptr_t)c2 % 16 == 0);
    return v4 ? launch_sum<float4>(partials, c, n1, kz1, p2, c2, n2, kz2, st) : launch_sum<float>(partials, c, n1, kz1, p2, c2, n2, kz2, st);
}

}  // namespace infr
