// Batched GEMM C[m, out_f] = Q8(x)[m, in_f] * W^T for Q4_K and Q6_K weights on tcgen05.mma kind::f16, exact in the
// integer block sums.
//
// Why f16 operands: every integer that the formats multiply is exactly representable in 11 bits, so the products and,
// while they stay below 2^24, their f32 sums are integers.  The operands are chosen so that every partial sum of a block does:
//   Q4_K  (q - 8) * sc    <= 8 * 63 = 504        one multiply per weight; an int8 form needs two (q * (sc & 7), q * (sc >> 3)).  A block's
//                                                 sum stays below 504 * 127 * 256 < 2^24 (q * sc: 3.1e7); the last instruction of a block
//                                                 adds 8 * sum_s sc_s * bsum_s (K = 16, as below): one rounding, where |sum| > 2^24.
//                                                 (All of it times 2^-14, which the row scale takes back: unpack_q4.)
//   Q4_K  m_s, 64h + l    the block minimum: sum_s m_s * bsum_s as ONE K = 16 instruction (8 sub-blocks x {64h, l})
//   Q6_K  sl * (q - 32), sh * (q - 32)            sc = 16 sh + sl, one accumulator each (a block's |L| <= 15 * 32 * 127 * 256 and |H|
//                                                 <= 8 * 32 * 127 * 256 stay below 2^24; sums of sc * (q - 32) reach 1.3e8); sum = 16 H + L
// The f32 expression of the CPU is applied per block (crates/infr-cpu/src/kernels.rs:151-184, :487-526):
// C += d8 * (d * sd - dmin * sm), C += (d8 * d) * sd, accumulated in block order in registers.
//
// Roles (one 128-row x TN-token tile at a time, persistent over tiles; a job = one block sum per output):
//   warps 0-7   unpack: thread = weight row; raw block -> f16 operand words -> TENSOR MEMORY (tcgen05.st) in slots of 32 columns
//               = 64 operand values, each published by itself; two teams (four warps = 128 rows) fill the two halves of a block
//   kEpi warps  epilogue: tensor-memory lane quarter x column part; folds a job's sums into running f32 registers
//   1 warp      block headers: row scales for the epilogue; Q4_K: minima and scales as operands of the two K = 16 instructions
//   1 producer  raw rows by tiled TMA (zero-filled past the matrix); a job's activation operands by two plain bulk copies (laid out
//               per token tile by gemm_tc_prep_kernel, so that they are contiguous)
//   2 issuers   in turn a job; one elected thread that runs the whole loop.  (A warp that runs the loop and issues under `lane == 0` spends 54
//               cycles on each tcgen05.mma, under an elect around a batch 20, a lone thread 8: clock64 around 8 instructions.)
// A raw stage is given back when it has been unpacked; what the epilogue needs of a block (row and token scales) has rings of its
// own, so that the weights' ring covers the memory's latency and not the whole pipeline's.
// TN = 32 (Q4_K) keeps to half an SM's shared and tensor memory, so that two CTAs hide each other's waits.
// Tiles: whole waves of them are multiplied over all of K; the rest of them is split over K so that it fills the SMs too, and a
// small kernel adds the parts in split order (deterministic).
// What bounds it: every role is a chain of dependent instructions and of barriers that cost its warp 100 to 200 cycles each, seen or not; a
// barrier between two roles is therefore as dear as what it guards.  Hence one barrier for a job's activation operands, none for giving them
// back where the accumulators' says as much, one epilogue warp that waits for the others (they stand at a named barrier), two issuers (one was
// busy for 2400 cycles of a job's 2550), and as few instructions as can be for a weight.  Q6_K's unpacking is the longest part of a job: nibble and high bits
// meet in one LOP3 before the bytes part, the offset is inside the multiply-add, rows are read in 8-byte words from a pitch of 240 bytes and
// the two teams' slots are multiplied in turn.  At 128 tokens a Q4_K job takes ~2320 cycles, its MMAs 1150; the warps issue 5980 instructions.
// Measured (B200, us, whole calls over rotated cold weights, back to back, so that a call's layout launch overlaps the call before):
//   Q4_K  4096 -> 14336  113 rows 26.8, 512 rows 74 (a call that waits for the one before it 86), 1024 rows 136;  14336 -> 4096, 1024 rows 150;  4096 -> 28672, 32 rows 31.6
//   Q6_K  14336 -> 4096  64 rows 37, 113 rows 43.1, 512 rows 136, 1000 rows 246;  4096 -> 14336  64 rows 37.8, 113 rows 45, 512 rows 125;  4096 -> 4096, 113 rows 20.2
// What the steps gave: one elected thread that issues, stages given back when unpacked, only the last tiles split over K: Q4_K, 512 rows 113 -> 82;
// the unpacking of Q6_K 4096 -> 14336, 64 rows 53 -> 42; Q6_K at 128 tokens in one pass (kJobBuf); fewer barriers, two issuers, nibbles as subnormals 82 -> 74 and
// Q6_K 14336 -> 4096, 512 rows 148 -> 142; Q6_K's waits (kFarWaits, the issuer's for the accumulators) 142 -> 136, and calls with a few jobs a CTA, which
// the step before had slowed down, 21.2 -> 20.2.
// Tried: 16 unpack and 8 epilogue warps (4 % slower), waits as tight loops in PTX (30 to 100 % slower: they poll more often), sleeping
// between polls (1 to 15 % slower), the issuer's loop not unrolled (17 % slower), a look at all of a job's barriers at once (no gain), a chunk's
// tensor-memory load during the fold of the one before it (spills).
// Every wait is bounded: on expiry the role raises a CTA flag and a status word, every role leaves its loop, copies in
// flight are drained and the tensor memory is freed.
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "f32x2.cuh"
#include "gemv_common.cuh"
#include "pdl.cuh"
#include "q8_code.cuh"
#include "row_norm.cuh"

namespace infr {
namespace {

constexpr int kTM = 128;
constexpr uint32_t kSpin = 1u << 22;
enum : int { F_Q4 = 0, F_Q6 = 1 };

template <int FMT, int TN>
struct Cfg {
    static constexpr int kUnits = FMT == F_Q4 ? 2 : 4;               // activation operands (two slots each) per job
    static constexpr int kUse = FMT == F_Q4 ? 2 : 4;                 // slots that a team fills per job
    static constexpr int kUnpack = 8;
    static constexpr int kAcc = FMT == F_Q4 ? 1 : 2;                 // accumulators per job
    // Jobs that have accumulators at a time.  Q6_K, 128 tokens: tensor memory holds those of one.  The operands of the next job are unpacked
    // while they are drained, so the drain costs nothing.  (Two passes of 64 tokens, one half drained while the other was multiplied, kept
    // every operand slot until the second pass: 14336 -> 4096, 113 rows 50.6 us, in one pass 46.9;
    // 1000 rows 296, 254.)
    static constexpr int kJobBuf = FMT == F_Q6 && TN == 128 ? 1 : 2;
    // Tensor memory that only one job has (Q4_K: the minima's sums) goes back as early as can be: Q4_K in a chain, 4096 -> 14336, 113 rows 28.8 ->
    // 28.5 us, 512 rows 80.0 -> 79.3, 14336 -> 4096, 1000 rows 171 -> 168; a call that waits for the one before it gains nothing (512 rows 90).
    // With two jobs' worth the fold is off the path: at 64 rows it cost 2 %.
    static constexpr bool kEarly = TN == 128;
    static constexpr int kRowBytes = FMT == F_Q6 ? 240 : 144;
    static constexpr int kRaw = kTM * kRowBytes;
    static constexpr int kUnitBytes = (FMT == F_Q4 ? 256 : 128) * TN;
    static constexpr int kExtra = FMT == F_Q4 ? 36 * TN : 4 * TN;    // per job: token scales, Q4_K also the split block sums
    // Slots of a team.  Each team of unpack warps owns its own: a team that shared one with another could find its barrier
    // two phases behind, which a parity wait cannot tell from "done".
    static constexpr int kSlots = FMT == F_Q4 && TN != 64 ? 2 : 4;
    static constexpr int kStages = TN == 64 || (FMT == F_Q6 && TN == 32) ? 4 : 3;
    static constexpr int kNB = FMT == F_Q6 ? 8 : (TN == 64 ? 6 : 4);
    static constexpr int kNX = 4;
    static constexpr int kMin = FMT == F_Q4 ? 2 * 4 * kTM * 16 : 0;  // two buffers of the minimum and the scale operand
    static constexpr int kRing = 4;                                  // row scales, per job
    static constexpr int kSmem = kNB * kUnitBytes + kStages * kRaw + kNX * kExtra + kMin + kRing * kTM * 4;
    static constexpr int kEpi = TN == 32 ? 4 : (TN == 128 ? 16 : 8);
    static constexpr int kCols = TN / (kEpi / 4);                    // output columns of an epilogue thread
    static constexpr int kChunk = TN == 64 && FMT == F_Q4 ? 16 : 8;  // columns per tensor-memory load (registers)
    static constexpr int W_HEAD = kUnpack + kEpi, W_LOAD = W_HEAD + 1, W_MMA = W_HEAD + 2, kWarps = W_HEAD + 4;
    static constexpr int kCtas = TN == 32 && FMT != F_Q6 ? 2 : 1;
    // The waits' loops as a function of their own.  Every role is at another place of the code, and with a loop at each wait Q6_K's warps lack an
    // instruction to issue more often (1.5 warps an issue slot, 1.4 this way): 1 us of a call with a few jobs a CTA.  us a call, loops at the
    // waits / one function: Q6_K 4096 -> 4096, 113 rows 21.2 / 20.35, 2048 -> 2048, 300 rows 19.6 / 18.5, 4096 -> 28672, 64 rows 71.6 / 65.9; Q4_K, whose
    // unpacking is shorter: 4096 -> 14336, 113 rows 27.6 / 28.4, 512 rows 75 / 77, 4096 -> 4096, 64 rows 13.5 / 13.7.
    static constexpr bool kFarWaits = FMT == F_Q6;
    // tensor-memory columns: accumulators of two jobs (one where there is no room), block-minimum sums of two jobs (one where there is no room), operands
    static constexpr int kMBuf = FMT == F_Q4 ? (TN == 128 ? 1 : 2) : 0;
    static constexpr uint32_t kColM = kJobBuf * kAcc * TN;
    static constexpr uint32_t kColA = kColM + kMBuf * TN;
    static constexpr uint32_t kCols0 = kColA + 2 * kSlots * 32;
    static constexpr uint32_t kTmem = kCols0 <= 256 ? 256 : 512;
    // barriers
    static constexpr int kJB = kNB / kUnits;                         // jobs whose activation operands fit
    static constexpr bool kOwnB = !(kJobBuf == 2 && kJB == 2);       // else B_ACCRDY says that a job's activation operands have been read
    static constexpr int B_SFULL = 0, B_SFREE = B_SFULL + kStages, B_XFULL = B_SFREE + kStages, B_XFREE = B_XFULL + kNX,
                         B_BFREE = B_XFREE + kNX, B_AFULL = B_BFREE + kJB, B_AFREE = B_AFULL + 4 * kUse, B_HEAD = B_AFREE + 2 * kSlots,
                         B_ACCRDY = B_HEAD + 2, B_ACCFREE = B_ACCRDY + 2, B_MFREE = B_ACCFREE + 2, B_DRAIN = B_MFREE + 1, B_COUNT = B_DRAIN + 2;
    static_assert(kCols0 <= 512 && (kCtas == 1 || kCols0 <= 256), "tensor memory");
    static_assert(kSmem <= (kCtas == 2 ? 111 : 226) * 1024, "shared memory");
    static_assert(kWarps <= 32 && kNB % kUnits == 0, "");
};

__device__ __forceinline__ uint32_t su32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// K-major operand without swizzle: planes of [rows][16 bytes], `lbo` bytes apart
__device__ __forceinline__ uint64_t mk_desc(uint32_t saddr, uint32_t lbo) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void mma_ta(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_sa(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tst32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]),
        "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tst_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tld(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tld(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

__device__ __forceinline__ bool try_bar(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Bounded wait; gives up early when another role has raised the CTA flag.  A role waits on a barrier by parity only where it
// has seen every earlier phase and the next completion depends on the waiter having passed, so it is never two phases off.
__device__ __forceinline__ bool poll_bar(uint32_t bar, uint32_t parity, volatile int *dead) {
    for (uint32_t i = 1; i < kSpin; i++) {
        if (try_bar(bar, parity)) return true;
        if ((i & 1023u) == 0 && *dead) return false;
    }
    return false;
}
__device__ __noinline__ bool poll_bar_far(uint32_t bar, uint32_t parity, volatile int *dead) { return poll_bar(bar, parity, dead); }
template <class K>
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int *dead) {
    if (try_bar(bar, parity)) return true;
    return K::kFarWaits ? poll_bar_far(bar, parity, dead) : poll_bar(bar, parity, dead);
}
// All lanes of a converged warp wait together: the result is one for the warp.
template <class K>
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int *dead) {
    return __all_sync(0xffffffffu, wait_bar<K>(bar, parity, dead));
}

// Named barrier 1 of N threads; true where `ok` is true in all of them.
template <int N>
__device__ __forceinline__ bool bar_and(bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.aligned.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r)
                 : "r"((uint32_t)ok), "n"(N)
                 : "memory");
    return r != 0;
}

__device__ __forceinline__ void tma2(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(map), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h2add(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ constexpr uint32_t dup(uint32_t h) { return h | (h << 16); }
// f16 bit patterns of the small constants used below (integers and powers of two)
constexpr uint32_t H_1024 = 0x6400, H_N1024 = 0xE400, H_N1152 = 0xE480, H_64 = 0x5400, H_N1032 = 0xE408, H_N1056 = 0xE420, H_2M14 = 0x0400,
                   H_N2M11 = 0x9000, H_NHALF = 0xB800;

// (a & m) | c in one instruction: with m and c in registers.  As constants they would be two immediates, which one LOP3 cannot take.
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t m, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(m), "r"(c));
    return r;
}
// the low nibbles of a's bytes under the high nibbles of b's
__device__ __forceinline__ uint32_t low_nibbles(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, 0x0F0F0F0F, 0xE4;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t in_reg(uint32_t v) {
    asm volatile("" : "+r"(v));
    return v;
}

// Q4_K: 64 elements = two sub-blocks in 8 words, scales s0 (low nibbles) and s1 (high nibbles); value = (q - 8) * scale * 2^-14.
// Operand values leave in the order (0, 2, 1, 3) of every four elements; gemm_tc_prep_kernel lays the activations out the same way.
// A nibble alone in a 16-bit half IS an f16: q * 2^-24 (subnormal) at bit 0, q * 2^-20 at bit 4.  With the scale times 2^10 and 2^6 one
// fused multiply-add gives q * sc * 2^-14 - 8 * sc * 2^-14, exact and not below the smallest normal: 9 instructions for 8 weights.  (A
// nibble under the f16 of 64, moved to bit 4, took 11: 4096 -> 28672 at 32 rows 33.0 -> 31.0 us, 512 rows of 4096 -> 14336 78.8 -> 76.7.)
__device__ __forceinline__ void unpack_q4(const uint32_t *w, uint32_t s0, uint32_t s1, uint32_t (&o)[32]) {
    const uint32_t t0 = h2add(dup(H_1024) | s0 * 0x10001u, dup(H_N1024)), t1 = h2add(dup(H_1024) | s1 * 0x10001u, dup(H_N1024));
    const uint32_t a0 = h2mul(t0, dup(H_1024)), a1 = h2mul(t1, dup(H_64)), c0 = h2mul(t0, dup(H_N2M11)), c1 = h2mul(t1, dup(H_N2M11));
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t v = w[i], x = v >> 8;
        o[2 * i] = h2fma(v & 0x000F000Fu, a0, c0);
        o[2 * i + 1] = h2fma(x & 0x000F000Fu, a0, c0);
        o[16 + 2 * i] = h2fma(v & 0x00F000F0u, a1, c1);
        o[17 + 2 * i] = h2fma(x & 0x00F000F0u, a1, c1);
    }
}

// Q6_K: 32 elements (part = 0..3 of a half block): low or high nibbles from ql[8 words], two high bits from qh[8 words], scales
// sc = 16 sh + sl of the two 16-element sub-blocks: bytes 2 (part & 1), + 1 of lw (sl, 0 <= sl < 16) and hw (sh + 8, -8 <= sh < 8).
// o[0..15] = sl * (q - 32), o[16..31] = sh * (q - 32), the same element order as above.  m = 0x003F003F, k = the f16 of 1024 twice (in_reg)
template <int PART>
__device__ __forceinline__ void unpack_q6(const uint32_t *ql, const uint32_t *qh, uint32_t lw, uint32_t hw, uint32_t m, uint32_t k, uint32_t (&o)[32]) {
#pragma unroll
    for (int g = 0; g < 2; g++) {
        constexpr uint32_t sel0 = 0x4040u + (PART & 1) * 0x0202u;  // the scale's byte below the high byte of the f16 of 1024, twice
        const uint32_t sl = h2add(__byte_perm(lw, 0x64646464u, sel0 + g * 0x0101u), dup(H_N1024));
        const uint32_t sh = h2add(__byte_perm(hw, 0x64646464u, sel0 + g * 0x0101u), dup(H_N1032));
        const uint32_t cl = h2mul(sl, dup(H_N1056)), ch = h2mul(sh, dup(H_N1056));  // (1024 + q) * s - 1056 * s: 33 * s has nine bits, one rounding, exact
#pragma unroll
        for (int i = 4 * g; i < 4 * g + 4; i++) {
            const uint32_t v = PART >= 2 ? ql[i] >> 4 : ql[i];
            const uint32_t y = PART == 0 ? qh[i] << 4 : PART == 1 ? qh[i] << 2 : PART == 2 ? qh[i] : qh[i] >> 2;
            const uint32_t q = low_nibbles(v, y), e = and_or(q, m, k), f = and_or(q >> 8, m, k);
            o[2 * i] = h2fma(e, sl, cl);
            o[2 * i + 1] = h2fma(f, sl, cl);
            o[16 + 2 * i] = h2fma(e, sh, ch);
            o[17 + 2 * i] = h2fma(f, sh, ch);
        }
    }
}

// N words from byte p + rem on, p 8-byte aligned, rem = 0, 2, 4 or 6
template <int N>
__device__ __forceinline__ void load_words(const uint8_t *p, int rem, uint32_t (&o)[N]) {
    static_assert(N % 2 == 0, "");
    uint32_t v[N + 2];
#pragma unroll
    for (int i = 0; i < N + 2; i += 2) {
        const uint2 w = *reinterpret_cast<const uint2 *>(p + 4 * i);
        v[i] = w.x, v[i + 1] = w.y;
    }
#pragma unroll
    for (int i = 0; i < N + 1; i++) v[i] = (rem & 4) ? v[i + 1] : v[i];
#pragma unroll
    for (int i = 0; i < N; i++) o[i] = __funnelshift_r(v[i], v[i + 1], (uint32_t)(rem & 2) * 8);
}

struct TcMat {
    float *c;  // [m, out_f]
    int out_f;
};
// Tiles [0, full) are multiplied over all of K; every other one by kz work items, whose parts [tile - full][split][TN][128 rows] go to
// `part` (kz == 1: straight to the result).
struct TcSplit {
    int full, kz;
    float *part;
};

}  // namespace

// Grouped (mixture-of-experts) form: the token dimension is a list of TN-token slabs, each holding up to TN activation rows
// routed to ONE expert; the weight rows of a slab's tiles are those of its expert inside the bank (experts back to back,
// out_f rows each) and its results go to the rows of its routed pairs.  slab_expert == nullptr: the plain GEMM.
struct TcGroup {
    const int *slab_expert;  // [n_slabs] expert (index inside the bank) of the slab
    const int *slab_p0;      // [n_slabs] first routed pair of the slab; output row = pair
    const int *slab_cnt;     // [n_slabs] pairs in the slab (1..TN)
    const int *n_slabs;      // device scalar
    const int *pair_row;     // [n_pairs] row of x of each pair (the layout of x)
};

namespace {

// Activations -> operand layout.  One warp per (token slot, 256 elements), or PER times 256, lane l owns elements [8l, 8l + 8) of them.
//   units:  [token tile][block][unit][plane][TN][16 B]  f16 codes, 8 per 16 bytes, in the order the unpack warps emit
//   extra:  [token tile][block]{Q4_K: [2][TN][8] f16 of 64h and l of the 32-element sums; scales [TN] f32}
// F32: quantises f32 rows (quantize_q8, crates/infr-cpu/src/quant.rs:27-58: the operations of quantize.cu in the same order);
// otherwise re-lays rows that are already quantised.  Slots past the last token are zero (grouped: as they were).
// PER > 1 (grouped): a slot's place in the work list is four dependent reads, and with a warp a block there are five waves of warps behind them
// (a layer of 256 rows over 128 experts, 2048 -> 768: 190.4 us one block a warp, 189.3; 200 rows over 16, 2048 -> 1024: 79.2, 76.6).
template <int FMT, bool F32, int PER>
__global__ void __launch_bounds__(256) gemm_tc_prep_kernel(const float *x, Q8Dev a, int m, int tn, int in_f, uint8_t *__restrict__ units,
                                                           uint8_t *__restrict__ extra, int n_tok, TcGroup grp) {
    pdl_go();
    pdl_wait();
    using C64 = Cfg<FMT, 64>;
    constexpr int UPS = C64::kUnits, UB = C64::kUnitBytes / 64, EB = C64::kExtra / 64;  // (per token: the same for every tile)
    const int lane = threadIdx.x & 31, nb = in_f >> 8;
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int per = (nb + PER - 1) / PER;  // warps of a slot
    if (wg >= (long long)n_tok * per) return;
    const int T = (int)(wg / per), b0 = (int)(wg % per) * PER, tt = T / tn, t = T - tt * tn;
    long long row = T < m ? T : -1;
    if (grp.slab_expert) {
        if (tt >= *grp.n_slabs) return;
        if (t >= grp.slab_cnt[tt]) return;  // (what a slot without a pair holds meets sums that are not stored: half the slots at 16 pairs an expert)
        row = grp.pair_row[grp.slab_p0[tt] + t];
    }
    float v[PER][8];
    uint2 c[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int b = b0 + k;
        c[k] = make_uint2(0, 0);
#pragma unroll
        for (int i = 0; i < 8; i++) v[k][i] = 0.f;
        if (row < 0 || b >= nb) continue;
        if (F32) {
            const float4 *xp = reinterpret_cast<const float4 *>(x + (size_t)row * in_f + (size_t)b * 256) + lane * 2;
            const float4 p = xp[0], q = xp[1];
            v[k][0] = p.x, v[k][1] = p.y, v[k][2] = p.z, v[k][3] = p.w, v[k][4] = q.x, v[k][5] = q.y, v[k][6] = q.z, v[k][7] = q.w;
        } else {
            c[k] = *reinterpret_cast<const uint2 *>(a.qs + (size_t)row * in_f + (size_t)b * 256 + lane * 8);
        }
    }
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int b = b0 + k;
        if (b >= nb) break;
        uint32_t w0 = 0, w1 = 0;  // eight codes
        float d = 0.f;
        int sum = 0;
        if (F32) {
            float am = 0.f;
#pragma unroll
            for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[k][i]));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
            d = am / 127.0f;
            const float id = d > 0.0f ? 1.0f / d : 0.0f;
            w0 = q8_codes4(make_float4(v[k][0], v[k][1], v[k][2], v[k][3]), id);
            w1 = q8_codes4(make_float4(v[k][4], v[k][5], v[k][6], v[k][7]), id);
        } else if (row >= 0) {
            w0 = c[k].x, w1 = c[k].y;
            d = a.d[(size_t)row * nb + b];
        }
        if (FMT == F_Q4) {
            sum = q8_sum4(w0) + q8_sum4(w1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        }
        // byte -> f16: 1024 + (code + 128) - 1152
        auto pair16 = [](uint32_t two) { return h2add(__byte_perm(two, 0x64646464u, 0x4140), dup(H_N1152)); };
        const uint32_t e0 = w0 ^ 0x80808080u, e1 = w1 ^ 0x80808080u;
        const uint4 o = make_uint4(pair16(__byte_perm(e0, 0, 0x0020)), pair16(__byte_perm(e0, 0, 0x0031)), pair16(__byte_perm(e1, 0, 0x0020)),
                                   pair16(__byte_perm(e1, 0, 0x0031)));
        constexpr int PL = FMT == F_Q4 ? 16 : 8;  // planes per unit
        const int unit = lane / PL, pl = lane % PL;
        const size_t rec = (size_t)tt * nb + b;
        *reinterpret_cast<uint4 *>(units + ((rec * UPS + unit) * UB + (size_t)pl * 16) * tn + (size_t)t * 16) = o;
        uint8_t *ex = extra + rec * EB * tn;
        if (FMT == F_Q4) {
            const int h = sum >> 6, l = sum & 63;
            uint32_t v = (uint32_t)__half_as_ushort(__int2half_rn(h * 64)) | ((uint32_t)__half_as_ushort(__int2half_rn(l)) << 16);
            const uint32_t nx = __shfl_down_sync(0xffffffffu, v, 4);
            if ((lane & 7) == 0) {
                *reinterpret_cast<uint32_t *>(ex + (size_t)t * 16 + (lane >> 3) * 4) = __byte_perm(v, nx, 0x5410);
                *reinterpret_cast<uint32_t *>(ex + (size_t)tn * 16 + (size_t)t * 16 + (lane >> 3) * 4) = __byte_perm(v, nx, 0x7632);
            }
            if (lane == 0) reinterpret_cast<float *>(ex + (size_t)tn * 32)[t] = d;
        } else {
            if (lane == 0) reinterpret_cast<float *>(ex)[t] = d;
        }
    }
}

// The same layout and quantiser for a block that a warp holds as lane l = elements 4l..4l+3 (v[0]) and 128+4l.. (v[1]): what the kernels
// below end with, so that a row which a norm or a gated activation has just formed needs no launch (and no read) of its own.
template <int FMT>
__device__ __forceinline__ void store_operand(const float4 (&v)[2], int T, int b, int nb, int tn, uint8_t *__restrict__ units, uint8_t *__restrict__ extra) {
    using C64 = Cfg<FMT, 64>;
    constexpr int UPS = C64::kUnits, UB = C64::kUnitBytes / 64, EB = C64::kExtra / 64, PL = FMT == F_Q4 ? 16 : 8;
    const int lane = threadIdx.x & 31, tt = T / tn, t = T - tt * tn;
    float am = 0.f;
#pragma unroll
    for (int h = 0; h < 2; h++) am = fmaxf(fmaxf(am, fmaxf(fabsf(v[h].x), fabsf(v[h].y))), fmaxf(fabsf(v[h].z), fabsf(v[h].w)));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float d = am / 127.0f, id = d > 0.0f ? 1.0f / d : 0.0f;
    auto pair16 = [](uint32_t two) { return h2add(__byte_perm(two, 0x64646464u, 0x4140), dup(H_N1152)); };
    const size_t rec = (size_t)tt * nb + b;
    uint8_t *ex = extra + rec * EB * tn;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t codes = q8_codes4(v[h], id), e = codes ^ 0x80808080u;
        const int p = h * 16 + (lane >> 1), unit = p / PL, pl = p % PL;  // 8 elements a plane: two lanes fill its 16 bytes
        *reinterpret_cast<uint2 *>(units + ((rec * UPS + unit) * UB + (size_t)pl * 16) * tn + (size_t)t * 16 + (lane & 1) * 8) =
            make_uint2(pair16(__byte_perm(e, 0, 0x0020)), pair16(__byte_perm(e, 0, 0x0031)));
        if (FMT == F_Q4) {
            int sum = q8_sum4(codes);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if ((lane & 7) == 0) {
                __half *hl = reinterpret_cast<__half *>(ex + (size_t)t * 16) + h * 4 + (lane >> 3);
                hl[0] = __int2half_rn((sum >> 6) * 64);
                hl[(size_t)tn * 8] = __int2half_rn(sum & 63);
            }
        }
    }
    if (lane == 0) reinterpret_cast<float *>(ex + (FMT == F_Q4 ? (size_t)tn * 32 : 0))[t] = d;
}

// RMSNorm (of a + b with ADD) and the layout in one launch: CTA = token slot; the scaled row also goes to dst.
template <int FMT, bool ADD>
__global__ void __launch_bounds__(1024) gemm_tc_norm_prep_kernel(const float *a, const float *b, float *sum_dst, const float *__restrict__ w, float *__restrict__ dst,
                                                                 float eps, int m, int tn, int in_f, uint8_t *__restrict__ units, uint8_t *__restrict__ extra) {
    __shared__ float s_part[32];
    const int lane = threadIdx.x & 31, T = blockIdx.x, nb = in_f >> 8;
    if (T >= m) {  // a slot past the last token: zeros
        pdl_go();
        pdl_wait();
        const float4 zero[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        for (int c = threadIdx.x >> 5; c < nb; c += blockDim.x >> 5) store_operand<FMT>(zero, T, c, nb, tn, units, extra);
        return;
    }
    rms_norm_row<ADD>(a, b, sum_dst, w, in_f, eps, T, s_part, [&](int c, const float4 (&v)[2]) {
#pragma unroll
        for (int h = 0; h < 2; h++) *reinterpret_cast<float4 *>(dst + (size_t)T * in_f + c * 256 + h * 128 + lane * 4) = v[h];
        store_operand<FMT>(v, T, c, nb, tn, units, extra);
    });
}

// silu(gate) * up and the layout in one launch: a warp per (token slot, block); the rows also go to dst (null: nowhere; it may be gate or up).
// Grouped: a slot's row is its routed pair.
template <int FMT>
__global__ void __launch_bounds__(256) gemm_tc_silu_prep_kernel(const float *gate, const float *up, float *dst, int m, int tn, int in_f, uint8_t *__restrict__ units,
                                                                uint8_t *__restrict__ extra, int n_tok, TcGroup grp) {
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x & 31, nb = in_f >> 8;
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wg >= (long long)n_tok * nb) return;
    const int T = (int)(wg / nb), b = (int)(wg % nb);
    long long row = T < m ? T : -1;
    if (grp.slab_expert) {
        const int tt = T / tn, t = T - tt * tn;
        if (tt >= *grp.n_slabs) return;
        if (t >= grp.slab_cnt[tt]) return;  // (as above)
        row = grp.slab_p0[tt] + t;
    }
    float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (row >= 0) {
        const size_t e = (size_t)row * in_f + (size_t)b * 256 + lane * 4;
        float4 g[2], u[2];
#pragma unroll
        for (int h = 0; h < 2; h++) g[h] = *reinterpret_cast<const float4 *>(gate + e + h * 128), u[h] = *reinterpret_cast<const float4 *>(up + e + h * 128);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            v[h] = make_float4(silu_mul(g[h].x, u[h].x), silu_mul(g[h].y, u[h].y), silu_mul(g[h].z, u[h].z), silu_mul(g[h].w, u[h].w));
            if (dst) *reinterpret_cast<float4 *>(dst + e + h * 128) = v[h];
        }
    }
    store_operand<FMT>(v, T, b, nb, tn, units, extra);
}

template <int FMT, int TN>
__global__ void __launch_bounds__(Cfg<FMT, TN>::kWarps * 32, Cfg<FMT, TN>::kCtas)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2, const uint8_t *units,
                   const uint8_t *extra, TcMat m1, TcMat m2, int m, int in_f, uint32_t *__restrict__ status, TcGroup grp, TcSplit split) {
    using K = Cfg<FMT, TN>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *bring = smem;
    uint8_t *raw0 = bring + K::kNB * K::kUnitBytes;
    uint8_t *ext0 = raw0 + K::kStages * K::kRaw;
    uint8_t *amin = ext0 + K::kNX * K::kExtra;                      // [2]{minima, 8 * scales}[2 planes][128][16 B]
    uint32_t *dring = reinterpret_cast<uint32_t *>(amin + K::kMin);  // [kRing][128]: f16 d (and dmin above it)
    __shared__ uint64_t bars[K::B_COUNT];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_dead;
    volatile int *dead = &s_dead;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nst = in_f / 256;
    pdl_go();
    if (tid == 0) {
        s_dead = 0;
        for (int i = 0; i < K::B_COUNT; i++) {
            int cnt = 1;
            if (i >= K::B_SFREE && i < K::B_XFULL) cnt = K::kUnpack + 1;
            if (i >= K::B_XFREE && i < K::B_BFREE) cnt = K::kEpi;
            if (i >= K::B_AFULL && i < K::B_AFREE) cnt = 4;  // [job's parity][team][use]: a barrier belongs to one issuer, who sees all of its phases
            if (i >= K::B_ACCFREE && i <= K::B_MFREE) cnt = K::kEpi;
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(&bars[i])), "r"(cnt));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_base_s)), "r"(K::kTmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    auto bar = [&](int i) { return su32(&bars[0]) + 8u * (uint32_t)i; };
    const int rt1 = (m1.out_f + kTM - 1) / kTM, row_tiles = rt1 + (m2.out_f + kTM - 1) / kTM;
    struct Tile {
        int rt, tt, b0, b1, part;  // part: index of the partial result, -1: none
    };
    // consecutive CTAs share a token tile; a K split's range of blocks is [b0, b1)
    auto tile_of = [&](int i) {
        Tile t;
        int r = i, ks = 0, kz = 1;
        t.part = -1;
        if (i >= split.full && split.kz > 1) {
            kz = split.kz;
            t.part = i - split.full;
            r = split.full + t.part / kz;
            ks = t.part % kz;
        }
        t.rt = r % row_tiles;
        t.tt = r / row_tiles;
        t.b0 = ks * nst / kz;
        t.b1 = (ks + 1) * nst / kz;
        return t;
    };
    auto n_items = [&]() {
        const int tiles = row_tiles * (grp.slab_expert ? *grp.n_slabs : (m + TN - 1) / TN);
        return tiles > split.full ? split.full + (tiles - split.full) * split.kz : tiles;
    };
    auto stage_x = [](int b) { return FMT == F_Q6 ? ((b * 210) & ~15) / 2 : b * 36; };  // tensor-map column of a block: 16-byte aligned
    auto fail = [&](uint32_t code) {
        if (!*dead) atomicExch(status, code);
        *dead = 1;
    };

    if (warp == K::W_LOAD) {
        // ------------------------------------------------------------------ weights, activation operands
        struct Jobs {  // the jobs of this CTA, one after the other
            int i, b;
            Tile t;
        };
        int n = 0;
        auto first = [&](Jobs &c) {
            c.i = blockIdx.x;
            if (c.i < n) c.t = tile_of(c.i), c.b = c.t.b0;
        };
        auto next = [&](Jobs &c) {
            if (++c.b == c.t.b1 && (c.i += gridDim.x) < n) c.t = tile_of(c.i), c.b = c.t.b0;
        };
        Jobs cw{};
        int jw = 0;
        auto load_w = [&]() {  // the next job's weights
            const int s = jw % K::kStages;
            const bool second = cw.t.rt >= rt1;
            const int row0 = (grp.slab_expert ? grp.slab_expert[cw.t.tt] * m1.out_f : 0) + (second ? cw.t.rt - rt1 : cw.t.rt) * kTM;
            expect_tx(bar(K::B_SFULL + s), K::kRaw);
            tma2(su32(raw0 + s * K::kRaw), second ? &map_w2 : &map_w, stage_x(cw.b), row0, bar(K::B_SFULL + s));
            jw++;
            next(cw);
        };
        // weights do not depend on the kernels before this one: the first stages are fetched before the wait
        if (lane == 0 && !grp.slab_expert) {
            n = n_items();
            first(cw);
            while (jw < K::kStages && cw.i < n) load_w();
        }
        __syncwarp();
        pdl_wait();
        if (lane == 0) {
            if (grp.slab_expert) {
                n = n_items();
                first(cw);
                while (jw < K::kStages && cw.i < n) load_w();
            }
            Jobs ca;
            first(ca);
            int js = 0;
            bool ok = true;
            for (; ca.i < n; js++, next(ca)) {
                const int x = js % K::kNX;
                const size_t rec = (size_t)ca.t.tt * nst + ca.b;
                if (js >= K::kNX && !(ok = wait_bar<K>(bar(K::B_XFREE + x), (uint32_t)((js / K::kNX - 1) & 1), dead))) break;
                if (js >= K::kJB) {  // the operands of the job that had the place before have been read
                    const int p = js - K::kJB;
                    if (!(ok = K::kOwnB ? wait_bar<K>(bar(K::B_BFREE + js % K::kJB), (uint32_t)(p / K::kJB) & 1u, dead)
                                        : wait_bar<K>(bar(K::B_ACCRDY + (p & 1)), (uint32_t)(p >> 1) & 1u, dead)))
                        break;
                }
                expect_tx(bar(K::B_XFULL + x), K::kExtra + K::kUnits * K::kUnitBytes);
                bulk(su32(bring + (js % K::kJB) * K::kUnits * K::kUnitBytes), units + rec * K::kUnits * K::kUnitBytes, K::kUnits * K::kUnitBytes, bar(K::B_XFULL + x));
                bulk(su32(ext0 + x * K::kExtra), extra + rec * K::kExtra, K::kExtra, bar(K::B_XFULL + x));
                // the job before is unpacked by the time that the one before that has been multiplied
                if (js >= 1 && cw.i < n) {
                    if (!(ok = wait_bar<K>(bar(K::B_SFREE + (js - 1) % K::kStages), (uint32_t)((js - 1) / K::kStages) & 1u, dead))) {
                        js++;
                        break;
                    }
                    load_w();
                }
            }
            if (!ok) fail(5u);
            if (*dead) {
                // copies in flight land before the CTA's shared memory is released
                for (int k = jw > K::kStages ? jw - K::kStages : 0; k < jw; k++)
                    for (uint32_t i = 0; i < (1u << 14) && !try_bar(bar(K::B_SFULL + k % K::kStages), (uint32_t)((k / K::kStages) & 1)); i++) {
                    }
                for (int k = js > K::kNX ? js - K::kNX : 0; k < js; k++)
                    for (uint32_t i = 0; i < (1u << 14) && !try_bar(bar(K::B_XFULL + k % K::kNX), (uint32_t)((k / K::kNX) & 1)); i++) {
                    }
            }
        }
    } else if (warp >= K::W_MMA) {
        // ------------------------------------------------------------------ MMA issuers, in turn a job: one thread, all of the loop
        const int me = warp - K::W_MMA;
        pdl_wait();
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
            const uint64_t bd0 = mk_desc(su32(bring), TN * 16);
            const int n = n_items();
            int j = 0;               // jobs of this CTA, over all tiles
            bool ok = true;
            for (int i = blockIdx.x; i < n && ok; i += gridDim.x) {
                const Tile t = tile_of(i);
                for (int b = t.b0; b < t.b1; b++, j++) {
                    const int s = j & 1;
                    if (s != me) continue;
                    const uint32_t jp = (uint32_t)(j >> 1) & 1u;
                    const int sa = K::kJobBuf == 2 ? s : 0;  // its accumulators
                    const uint32_t q = (uint32_t)(j % K::kJB);  // its place in the activation ring
                    const uint32_t td = tmem + (uint32_t)(sa * K::kAcc * TN);
                    // what the header warp has seen: its own operands, and the accumulators given back by the job before last
                    if (!(ok = wait_bar<K>(bar(K::B_HEAD + s), jp, dead))) break;
                    if (!(ok = wait_bar<K>(bar(K::B_XFULL + j % K::kNX), (uint32_t)(j / K::kNX) & 1u, dead))) break;
                    // One job's accumulators: the other issuer's job gives them back (the one before that has, or B_HEAD would not be here, and its own
                    // barrier is the next to complete).  By the header warp, as where two jobs have some, it is a barrier more between the fold and the next
                    // product: 4096 -> 4096, 113 rows 20.35 / 20.2 us, 14336 -> 4096, 113 rows 44.8 / 43.7, 512 rows 142 / 136.
                    if (K::kJobBuf == 1 && j >= 1 && !(ok = wait_bar<K>(bar(K::B_ACCFREE + (s ^ 1)), (uint32_t)((j - 1) >> 1) & 1u, dead))) break;
#pragma unroll
                    for (int st = 0; st < 2 * K::kUnits; st++) {
                        // (Q6_K: the teams' slots in turn, both get theirs back early)
                        const int k8 = K::kUnits == 4 ? (st >> 2) * 2 + ((st >> 1) & 1) * 4 + (st & 1) : st;
                        const int u = k8 >> 1, h = k8 & 1, team = k8 / K::kUse;
                        const uint64_t bd = bd0 + (uint64_t)((q * K::kUnits + u) * (uint32_t)(K::kUnitBytes / 16));
                        const int sl = team * K::kSlots + (j * K::kUse + k8 % K::kUse) % K::kSlots;
                        if (!(ok = wait_bar<K>(bar(K::B_AFULL + (s * 2 + team) * K::kUse + k8 % K::kUse), jp, dead))) break;
                        tc_fence_after();
                        const uint32_t ta = tmem + K::kColA + (uint32_t)(sl * 32);
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            // Q6_K: the sl and the sh operands of a slot meet the same 32 activations
                            const int pl = FMT == F_Q6 ? h * 4 + (k & 1) * 2 : h * 8 + k * 2;
                            const uint32_t keep = (uint32_t)(st > 0 || (K::kAcc == 2 ? (k & 1) : k > 0));
                            mma_ta(td + (uint32_t)(K::kAcc == 2 ? (k >> 1) * TN : 0), ta + (uint32_t)(k * 8), bd + (uint64_t)(pl * TN), idesc, keep);
                        }
                        mma_commit(bar(K::B_AFREE + sl));
                    }
                    if (!ok) break;
                    if (FMT == F_Q4) {
                        const uint64_t xd = mk_desc(su32(ext0 + (j % K::kNX) * K::kExtra), TN * 16);
                        mma_sa(td, mk_desc(su32(amin + (s * 4 + 2) * kTM * 16), kTM * 16), xd, idesc, 1u);
                        // (the other issuer's job; the one before that is folded, or B_HEAD would not be here)
                        if (K::kMBuf == 1 && j >= 1 && !(ok = wait_bar<K>(bar(K::B_MFREE), (uint32_t)((j - 1) & 1), dead))) break;
                        tc_fence_after();
                        mma_sa(tmem + K::kColM + (uint32_t)(K::kMBuf == 2 ? s * TN : 0), mk_desc(su32(amin + s * 4 * kTM * 16), kTM * 16), xd, idesc, 0u);
                    }
                    if (K::kOwnB) mma_commit(bar(K::B_BFREE + q));
                    mma_commit(bar(K::B_ACCRDY + sa));
                }
            }
            if (!ok) fail(6u);
            // every issued MMA has completed before the tensor memory is freed
            mma_commit(bar(K::B_DRAIN + me));
            for (uint32_t i = 0; i < (1u << 20) && !try_bar(bar(K::B_DRAIN + me), 0u); i++) {
            }
        }
        __syncwarp();
    } else if (warp == K::W_HEAD) {
        // ------------------------------------------------------------------ block headers: lane = four rows
        pdl_wait();
        const int n = n_items();
        int js = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < n && ok; i += gridDim.x) {
            const Tile t = tile_of(i);
            for (int b = t.b0; b < t.b1; b++, js++) {
                const int ls = js % K::kStages, s = js & 1;
                if (!(ok = wait_warp<K>(bar(K::B_SFULL + ls), (uint32_t)((js / K::kStages) & 1), dead))) break;
                const uint8_t *blk = raw0 + ls * K::kRaw;
                uint4 hdr[4];
                uint32_t dh[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint8_t *r = blk + (size_t)(k * 32 + lane) * K::kRowBytes;
                    if (FMT == F_Q4)
                        hdr[k] = *reinterpret_cast<const uint4 *>(r), dh[k] = hdr[k].x;
                    else
                        dh[k] = *reinterpret_cast<const unsigned short *>(r + 208 + ((b * 210) & 15));
                }
                __syncwarp();
                if (lane == 0) bar_arrive(bar(K::B_SFREE + ls));
                // The job before last has been multiplied and its accumulators are given back: the rings' places are free (and where two jobs have
                // accumulators the issuer, who waits for this warp, need not wait for them).
                if (js >= 2 && !(ok = wait_warp<K>(bar(K::B_ACCFREE + s), (uint32_t)(((js >> 1) - 1) & 1), dead))) break;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    dring[(js % K::kRing) * kTM + k * 32 + lane] = dh[k];
                    if (FMT == F_Q4) {
                        const uint4 h = hdr[k];
                        const uint32_t n0 = h.z & 0x3F3F3F3Fu, n1 = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
                        const uint32_t c0 = h.y & 0x3F3F3F3Fu, c1 = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
                        auto two = [](uint32_t v, uint32_t sel) { return h2add(__byte_perm(v, 0x64646464u, sel), dup(H_N1024)); };
                        auto two8 = [](uint32_t v, uint32_t sel) { return h2fma(__byte_perm(v, 0x70707070u, sel), dup(H_2M14), dup(H_NHALF)); };  // 8 v * 2^-14
                        const uint4 p = make_uint4(two(n0, 0x4140), two(n0, 0x4342), two(n1, 0x4140), two(n1, 0x4342));
                        const uint4 e = make_uint4(two8(c0, 0x4140), two8(c0, 0x4342), two8(c1, 0x4140), two8(c1, 0x4342));
                        uint4 *mp = reinterpret_cast<uint4 *>(amin + s * 4 * kTM * 16) + k * 32 + lane;
                        mp[0] = p;
                        mp[kTM] = p;
                        mp[2 * kTM] = e;
                        mp[3 * kTM] = e;
                    }
                }
                if (FMT == F_Q4) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(bar(K::B_HEAD + s));
            }
        }
        if (!ok) fail(7u);
    } else if (warp < K::kUnpack) {
        // ------------------------------------------------------------------ unpack warps
        pdl_wait();
        const int n = n_items();
        const int quarter = warp & 3, team = warp >> 2, row = quarter * 32 + lane;
        const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16) + K::kColA;
        const uint32_t km = in_reg(0x003F003Fu), kc = in_reg(dup(H_1024));  // (Q6_K)
        int js = 0;
        bool ok = true;
        // the team's slot of its use-th operand run: its previous MMAs are complete, it is filled, it is announced
        auto put = [&](int use, const uint32_t (&o)[32]) {
            const int sl = team * K::kSlots + use % K::kSlots, ph = use / K::kSlots;
            if (ph >= 1 && !wait_warp<K>(bar(K::B_AFREE + sl), (uint32_t)((ph - 1) & 1), dead)) return false;
            tc_fence_after();
            tst32(tl + (uint32_t)(sl * 32), o);
            tst_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(bar(K::B_AFULL + ((use / K::kUse & 1) * 2 + team) * K::kUse + use % K::kUse));
            return true;
        };
        for (int i = blockIdx.x; i < n && ok; i += gridDim.x) {
            const Tile t = tile_of(i);
            for (int b = t.b0; b < t.b1; b++, js++) {
                const int ls = js % K::kStages;
                if (!(ok = wait_warp<K>(bar(K::B_SFULL + ls), (uint32_t)((js / K::kStages) & 1), dead))) break;
                const uint8_t *blk = raw0 + ls * K::kRaw + (size_t)row * K::kRowBytes;
                const uint4 *bv = reinterpret_cast<const uint4 *>(blk);
                uint32_t o[32];
                auto given_back = [&]() {
                    __syncwarp();
                    if (lane == 0) bar_arrive(bar(K::B_SFREE + ls));
                };
                if (FMT == F_Q4) {
                    const uint4 hdr = bv[0];
                    const uint4 q0 = bv[1 + 4 * team], q1 = bv[2 + 4 * team], q2 = bv[3 + 4 * team], q3 = bv[4 + 4 * team];
                    const uint32_t w[16] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, q3.x, q3.y, q3.z, q3.w};
                    const uint32_t sc = team ? (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u) : hdr.y & 0x3F3F3F3Fu;
                    given_back();
                    unpack_q4(w, sc & 0xFFu, (sc >> 8) & 0xFFu, o);
                    if (!(ok = put(js * 2, o))) break;
                    unpack_q4(w + 8, (sc >> 16) & 0xFFu, sc >> 24, o);
                    if (!(ok = put(js * 2 + 1, o))) break;
                } else {
                    // half block `team`: the low and then the high nibbles of its 64 bytes
                    const int off = (b * 210) & 15, rem = off & 7;
                    const uint8_t *p = blk + (off & 8);
                    uint32_t ql[16], qh[8], sc[2];
                    load_words(p + 64 * team, rem, ql);
                    load_words(p + 128 + 32 * team, rem, qh);
                    load_words(p + 192 + 8 * team, rem, sc);
                    given_back();
                    const uint32_t l0 = sc[0] & 0x0F0F0F0Fu, l1 = sc[1] & 0x0F0F0F0Fu;
                    const uint32_t h0 = ((sc[0] >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u, h1 = ((sc[1] >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
                    unpack_q6<0>(ql, qh, l0, h0, km, kc, o);
                    if (!(ok = put(js * 4, o))) break;
                    unpack_q6<1>(ql + 8, qh, l0, h0, km, kc, o);
                    if (!(ok = put(js * 4 + 1, o))) break;
                    unpack_q6<2>(ql, qh, l1, h1, km, kc, o);
                    if (!(ok = put(js * 4 + 2, o))) break;
                    unpack_q6<3>(ql + 8, qh, l1, h1, km, kc, o);
                    if (!(ok = put(js * 4 + 3, o))) break;
                }
            }
        }
        if (!ok) fail(7u);
    } else {
        // ------------------------------------------------------------------ epilogue warps
        pdl_wait();
        const int n = n_items();
        const int quarter = warp & 3, part = (warp - K::kUnpack) >> 2, row = quarter * 32 + lane, col0 = part * K::kCols;
        const uint32_t tlane = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
        u64 acc[K::kCols / 2];  // pairs of columns
        int j = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < n && ok; i += gridDim.x) {
            const Tile t = tile_of(i);
#pragma unroll
            for (int k = 0; k < K::kCols / 2; k++) acc[k] = 0ull;
#pragma unroll 1
            for (int b = t.b0; b < t.b1; b++, j++) {
                const int x = j % K::kNX, s = K::kJobBuf == 2 ? j & 1 : 0;
                // one warp waits (sixteen of them took 1500 instructions a job to look, Q6_K at 512 rows 148 -> 141 us), the others stand at the barrier
                if (warp == K::kUnpack)
                    ok = wait_bar<K>(bar(K::B_XFULL + x), (uint32_t)((j / K::kNX) & 1), dead) &&
                         wait_bar<K>(bar(K::B_ACCRDY + s), (uint32_t)((K::kJobBuf == 2 ? j >> 1 : j) & 1), dead);
                __syncwarp();
                if (!(ok = bar_and<K::kEpi * 32>(ok))) break;
                tc_fence_after();
                const float *d8 = reinterpret_cast<const float *>(ext0 + x * K::kExtra + (FMT == F_Q4 ? 32 * TN : 0)) + col0;
                const uint32_t hd = dring[(j % K::kRing) * kTM + row];
                const u64 dw = f2_dup(FMT == F_Q4 ? h2f(hd) * 16384.f : h2f(hd)), nm = f2_dup(FMT == F_Q4 ? -h2f(hd >> 16) : 16.f);
                auto give_back = [&]() {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (K::kMBuf == 1) bar_arrive(bar(K::B_MFREE));  // before ACCFREE: an issuer that saw that one is one phase behind at most
                        bar_arrive(bar(K::B_ACCFREE + (j & 1)));
                    }
                };
#pragma unroll
                for (int c = 0; c < K::kCols; c += K::kChunk) {
                    uint32_t sd[K::kChunk], sm[K::kChunk];
                    tld(tlane + (uint32_t)(s * K::kAcc * TN + c), sd);
                    if (FMT == F_Q4) tld(tlane + K::kColM + (uint32_t)((K::kMBuf == 2 ? s * TN : 0) + c), sm);
                    if (K::kAcc == 2) tld(tlane + (uint32_t)(s * K::kAcc * TN + TN + c), sm);
                    tld_wait();
                    // all of the job is in registers: its accumulators go back before the last chunk is folded
                    if (K::kEarly && c + K::kChunk == K::kCols) give_back();
#pragma unroll
                    for (int k4 = 0; k4 < K::kChunk / 4; k4++) {
                        const ulonglong2 dv = *reinterpret_cast<const ulonglong2 *>(d8 + c + 4 * k4);
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const int e = 4 * k4 + 2 * k, a = (c + e) / 2;
                            const u64 f = f2_pack(sd[e], sd[e + 1]), g = f2_pack(sm[e], sm[e + 1]), d = k ? dv.y : dv.x;
                            if (FMT == F_Q4)
                                acc[a] = f2_fma(d, f2_fma(nm, g, f2_mul(dw, f)), acc[a]);
                            else
                                acc[a] = f2_fma(f2_mul(dw, d), f2_fma(nm, g, f), acc[a]);
                        }
                    }
                }
                if (!K::kEarly) give_back();
                __syncwarp();
                if (lane == 0) bar_arrive(bar(K::B_XFREE + x));
            }
            if (!ok) break;
            auto val = [&](int k) { return __uint_as_float((uint32_t)(acc[k / 2] >> (32 * (k & 1)))); };
            if (t.part >= 0) {
                float *P = split.part + ((size_t)t.part * TN + col0) * kTM + row;
#pragma unroll
                for (int k = 0; k < K::kCols; k++) P[k * kTM] = val(k);
            } else {
                const bool second = t.rt >= rt1;
                const int of = second ? m2.out_f : m1.out_f;
                const int grow = (second ? t.rt - rt1 : t.rt) * kTM + row;
                const int lim = grp.slab_expert ? grp.slab_cnt[t.tt] : m - t.tt * TN;
                const size_t orow = grp.slab_expert ? (size_t)grp.slab_p0[t.tt] : (size_t)t.tt * TN;
                float *C = (second ? m2.c : m1.c) + orow * of + grow;
                if (grow < of) {
#pragma unroll
                    for (int k = 0; k < K::kCols; k++)
                        if (col0 + k < lim) C[(size_t)(col0 + k) * of] = val(k);
                }
            }
            __syncwarp();
        }
        if (!ok) fail(4u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(K::kTmem));
}

// The parts of the tiles that are split over K, added in split order (the same bits on every run).  Block = 8 tokens x 128 rows of a
// tile, a warp one token.
__global__ void __launch_bounds__(256) gemm_tc_sum_kernel(TcSplit split, TcMat m1, TcMat m2, int m, int tn) {
    pdl_go();
    pdl_wait();
    const int per = tn / 8, ti = blockIdx.x / per, tok = (blockIdx.x % per) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int rt1 = (m1.out_f + kTM - 1) / kTM, row_tiles = rt1 + (m2.out_f + kTM - 1) / kTM;
    const int r = split.full + ti, rt = r % row_tiles, tt = r / row_tiles;
    if (tt * tn + tok >= m) return;
    const float4 *p = reinterpret_cast<const float4 *>(split.part + ((size_t)ti * split.kz * tn + tok) * kTM) + lane;
    float4 a = p[0];
#pragma unroll 4
    for (int k = 1; k < split.kz; k++) {
        const float4 v = p[(size_t)k * tn * (kTM / 4)];
        a.x += v.x, a.y += v.y, a.z += v.z, a.w += v.w;
    }
    const bool second = rt >= rt1;
    const int of = second ? m2.out_f : m1.out_f, grow = (second ? rt - rt1 : rt) * kTM + lane * 4;
    float *C = (second ? m2.c : m1.c) + (size_t)(tt * tn + tok) * of + grow;
    const float v[4] = {a.x, a.y, a.z, a.w};
    if (grow + 4 <= of && ((uintptr_t)C & 15) == 0) {
        *reinterpret_cast<float4 *>(C) = a;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (grow + k < of) C[k] = v[k];
    }
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                             const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

int fmt_of(int dtype) { return dtype == DT_Q4K ? F_Q4 : F_Q6; }
size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// Activation layout sizes for `n_tok` slots (a multiple of the token tile).
size_t units_bytes(int n_tok, int in_f) { return align256((size_t)n_tok * (in_f / 256) * 512); }
size_t extra_bytes(int fmt, int n_tok, int in_f) { return align256((size_t)n_tok * (in_f / 256) * (fmt == F_Q4 ? 36 : 4)); }

bool weight_map(int fmt, const uint8_t *w, size_t rows, int in_f, CUtensorMap *map) {
    EncodeFn enc = encode_fn();
    if (!enc) return false;
    const cuuint32_t one2[2] = {1, 1};
    if (fmt == F_Q6) {
        const cuuint64_t nb = (cuuint64_t)in_f / 256, gdim[2] = {nb * 105, (cuuint64_t)rows}, gstr[1] = {nb * 210};
        const cuuint32_t box[2] = {Cfg<F_Q6, 128>::kRowBytes / 2, kTM};
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<uint8_t *>(w), gdim, gstr, box, one2, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
    const cuuint64_t rb = (cuuint64_t)(in_f / 256) * 144, gdim[2] = {rb / 4, (cuuint64_t)rows}, gstr[1] = {rb};
    const cuuint32_t box[2] = {36, kTM};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t *>(w), gdim, gstr, box, one2, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int FMT, int TN>
cudaError_t launch_fmt(const CUtensorMap &mw, const CUtensorMap &mw2, const uint8_t *units, const uint8_t *extra, TcMat m1, TcMat m2, int m, int in_f,
                       uint32_t *status, const TcGroup &grp, const TcSplit &split, int grid, cudaStream_t st) {
    using K = Cfg<FMT, TN>;
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<FMT, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, K::kSmem);
    if (e != cudaSuccess) return e;
    return launch_pdl(gemm_tc_kernel<FMT, TN>, dim3((unsigned)grid), dim3(K::kWarps * 32), (size_t)K::kSmem, st, mw, mw2, units, extra, m1, m2, m, in_f,
                      status, grp, split);
}

template <int FMT>
cudaError_t launch_tn(int tn, const CUtensorMap &mw, const CUtensorMap &mw2, const uint8_t *units, const uint8_t *extra, TcMat m1, TcMat m2, int m,
                      int in_f, uint32_t *status, const TcGroup &grp, const TcSplit &split, int grid, cudaStream_t st) {
    if (tn == 32) return launch_fmt<FMT, 32>(mw, mw2, units, extra, m1, m2, m, in_f, status, grp, split, grid, st);
    if (tn == 64) return launch_fmt<FMT, 64>(mw, mw2, units, extra, m1, m2, m, in_f, status, grp, split, grid, st);
    return launch_fmt<FMT, 128>(mw, mw2, units, extra, m1, m2, m, in_f, status, grp, split, grid, st);
}

constexpr int kGroupedPer = 2;  // blocks of a warp, grouped
template <bool F32>
cudaError_t launch_prep(int fmt, const float *x, const Q8Dev &a, int m, int tn, int in_f, uint8_t *units, uint8_t *extra, int n_tok, const TcGroup &grp,
                        cudaStream_t st) {
    const int nb = in_f / 256, per = grp.slab_expert ? (nb + kGroupedPer - 1) / kGroupedPer : nb;
    const dim3 grid((unsigned)(((size_t)n_tok * per + 7) / 8)), block(256);
    if constexpr (F32)
        if (grp.slab_expert) return launch_pdl(gemm_tc_prep_kernel<F_Q4, F32, kGroupedPer>, grid, block, 0, st, x, a, m, tn, in_f, units, extra, n_tok, grp);
    if (fmt == F_Q4) return launch_pdl(gemm_tc_prep_kernel<F_Q4, F32, 1>, grid, block, 0, st, x, a, m, tn, in_f, units, extra, n_tok, grp);
    return launch_pdl(gemm_tc_prep_kernel<F_Q6, F32, 1>, grid, block, 0, st, x, a, m, tn, in_f, units, extra, n_tok, grp);
}

int ctas_of(int fmt, int tn, const DeviceInfo &dev) { return dev.sm_count * (tn == 32 && fmt != F_Q6 ? 2 : 1); }

// How the tiles go to the CTAs.
// One token tile (up to 128 rows): every tile's K is split kz ways (a batch of a few dozen rows against a matrix with few row tiles
// would otherwise keep most SMs idle).  The split decides the order of a result's f32 additions, and between the layers of a model
// values are coded in 8 bits, where another order moves codes: the constants of this estimate (microseconds a block of a tile, 2 a
// tile's start and end, 2.5 the kernel that adds the parts, 2e-6 each of their words) stay what they were, so that a decode step or a
// prompt chunk keeps its bits.  They are high by a quarter by now; with others 113 rows of 4096 -> 14336 took the same time.
// More tokens: whole waves of tiles (or all but one of them) are not split, the remaining ones fill the SMs (448 tiles on 148 SMs: 3 waves,
// and 4 tiles over 8 CTAs each).  Estimate in microseconds: blk a block of a tile, tile its start and end, sum the kernel that adds the
// parts, word each of their words; fitted to 130..1024 rows of 13 shapes with up to 23 splits each, where the choice is 1.2 % (Q4_K) and
// 0.1 % (Q6_K) above the best of them on average, 10 % and 2 % at worst.  (Q6_K, 130 rows of 4096 -> 5120: 54 us unsplit, 46 three ways.)
TcSplit split_of(int fmt, int tn, int m, int in_f, int row_tiles, int out_f, const DeviceInfo &dev) {
    const int cap = ctas_of(fmt, tn, dev), tt = (m + tn - 1) / tn, tiles = row_tiles * tt, nst = in_f / 256;
    if (tt == 1) {
        const int n_tiles = (out_f + kTM - 1) / kTM;  // (of both heights together)
        const double stage = fmt == F_Q4 ? (tn == 128 ? 1.5 : 1.2) : 2.5;
        int best = 1;
        double best_cost = 1e30;
        for (int kz = 1; kz <= 16 && kz <= nst; kz++) {
            const int waves = (n_tiles * kz + cap - 1) / cap, len = (nst + kz - 1) / kz;
            const double cost = waves * (len * stage + 2.0) + (kz > 1 ? 2.5 + 2e-6 * kz * m * (double)out_f : 0.0);
            if (cost < best_cost * 0.98) best = kz, best_cost = cost;
        }
        return best == 1 ? TcSplit{tiles, 1, nullptr} : TcSplit{0, best, nullptr};
    }
    const bool q4 = fmt == F_Q4;
    const double blk = q4 ? 1.2 : 2.7, tile = q4 ? 3.0 : 2.0, sum = q4 ? 1.5 : 2.0, word = q4 ? 1e-6 : 2e-7;
    TcSplit best{tiles, 1, nullptr};
    double best_cost = (double)((tiles + cap - 1) / cap) * (nst * blk + tile);
    for (int full = tiles / cap * cap, k = 0; k < 2 && full >= 0; k++, full -= cap) {
        const int rest = tiles - full;
        for (int kz = 2; kz <= 16 && kz <= nst && rest > 0; kz++) {
            const int waves = (rest * kz + cap - 1) / cap, len = (nst + kz - 1) / kz;
            const double cost = (double)(full / cap) * (nst * blk + tile) + waves * (len * blk + tile) + sum + word * rest * kz * tn * kTM;
            if (cost < best_cost * 0.98) best = TcSplit{full, kz, nullptr}, best_cost = cost;
        }
    }
    return best;
}
size_t part_bytes(const TcSplit &s, int tiles, int tn) { return s.kz > 1 ? (size_t)(tiles - s.full) * s.kz * tn * kTM * 4 : 0; }

}  // namespace

// Rows the tiled copies can fetch: whole blocks, row bytes a multiple of 16.
bool gemm_tc_takes(int dtype, int in_f) {
    if (in_f <= 0) return false;
    if (dtype == DT_Q4K) return in_f % 256 == 0;
    return dtype == DT_Q6K && in_f % 2048 == 0;
}

// Token tile for a batch of m rows.  It depends on m alone, so that Linears of one format on the same rows share the layout.
static int tile_of_batch(int m) { return m <= 32 ? 32 : (m <= 64 ? 64 : 128); }

size_t gemm_tc_record_bytes(int dtype, int m, int in_f) {
    const int tn = tile_of_batch(m), n = (m + tn - 1) / tn * tn;
    return units_bytes(n, in_f) + extra_bytes(fmt_of(dtype), n, in_f);
}

static int row_tiles_of(int out_f1, int out_f2) { return (out_f1 + kTM - 1) / kTM + (out_f2 + kTM - 1) / kTM; }
size_t gemm_tc_partial_bytes(int dtype, int m, int in_f, int out_f1, int out_f2, const DeviceInfo &dev) {
    const int tn = tile_of_batch(m), rt = row_tiles_of(out_f1, out_f2);
    return part_bytes(split_of(fmt_of(dtype), tn, m, in_f, rt, out_f1 + out_f2, dev), rt * ((m + tn - 1) / tn), tn);
}

cudaError_t launch_gemm_tc_prep(int dtype, const float *x, const Q8Dev *a, void *records, int m, int in_f, cudaStream_t st) {
    if (m < 1 || !gemm_tc_takes(dtype, in_f) || (x && ((uintptr_t)x % 16))) return cudaErrorInvalidValue;
    const int f = fmt_of(dtype), tn = tile_of_batch(m), n = (m + tn - 1) / tn * tn;
    uint8_t *u = static_cast<uint8_t *>(records), *e = u + units_bytes(n, in_f);
    return x ? launch_prep<true>(f, x, Q8Dev{}, m, tn, in_f, u, e, n, TcGroup{}, st) : launch_prep<false>(f, nullptr, *a, m, tn, in_f, u, e, n, TcGroup{}, st);
}

// The same from what forms the rows (RowSource).
cudaError_t launch_gemm_tc_prep(int dtype, const RowSource &src, void *records, int m, int in_f, cudaStream_t st) {
    if (m < 1 || !gemm_tc_takes(dtype, in_f)) return cudaErrorInvalidValue;
    const int f = fmt_of(dtype), tn = tile_of_batch(m), n = (m + tn - 1) / tn * tn, nb = in_f / 256;
    uint8_t *u = static_cast<uint8_t *>(records), *e = u + units_bytes(n, in_f);
    if (!src.norm_w) {
        auto kernel = f == F_Q4 ? gemm_tc_silu_prep_kernel<F_Q4> : gemm_tc_silu_prep_kernel<F_Q6>;
        return launch_pdl(kernel, dim3((unsigned)(((size_t)n * nb + 7) / 8)), dim3(256), 0, st, src.a, src.b, src.dst, m, tn, in_f, u, e, n, TcGroup{});
    }
    const int threads = nb > 32 ? 1024 : nb * 32;
    auto kernel = f == F_Q4 ? (src.b ? gemm_tc_norm_prep_kernel<F_Q4, true> : gemm_tc_norm_prep_kernel<F_Q4, false>)
                            : (src.b ? gemm_tc_norm_prep_kernel<F_Q6, true> : gemm_tc_norm_prep_kernel<F_Q6, false>);
    return launch_pdl(kernel, dim3((unsigned)n), dim3((unsigned)threads), 0, st, src.a, src.b, src.sum, src.norm_w, src.dst, src.eps, m, tn, in_f, u, e);
}

cudaError_t launch_gemm_tc(int dtype, const uint8_t *w, const void *records, float *c, float *partials, int m, int in_f, int out_f, const DeviceInfo &dev,
                           uint32_t *status, cudaStream_t st, const uint8_t *w2, float *c2, int out_f2) {
    if (m < 1 || out_f < 1 || !gemm_tc_takes(dtype, in_f)) return cudaErrorInvalidValue;
    if (!w2) out_f2 = 0;
    const int f = fmt_of(dtype), tn = tile_of_batch(m), tt = (m + tn - 1) / tn, n = tt * tn;
    const uint8_t *u = static_cast<const uint8_t *>(records), *e = u + units_bytes(n, in_f);
    const int rt = row_tiles_of(out_f, out_f2), tiles = rt * tt;
    TcSplit split = split_of(f, tn, m, in_f, rt, out_f + out_f2, dev);
    if (split.kz > 1 && !partials) return cudaErrorInvalidValue;
    split.part = partials;
    CUtensorMap mw, mw2;
    if (!weight_map(f, w, (size_t)out_f, in_f, &mw)) return cudaErrorInvalidValue;
    mw2 = mw;
    if (w2 && !weight_map(f, w2, (size_t)out_f2, in_f, &mw2)) return cudaErrorInvalidValue;
    const TcMat m1{c, out_f}, m2{c2, out_f2};
    const int items = split.full + (tiles - split.full) * split.kz, cap = ctas_of(f, tn, dev), grid = items < cap ? items : cap;
    cudaError_t r = f == F_Q4 ? launch_tn<F_Q4>(tn, mw, mw2, u, e, m1, m2, m, in_f, status, TcGroup{}, split, grid, st)
                              : launch_tn<F_Q6>(tn, mw, mw2, u, e, m1, m2, m, in_f, status, TcGroup{}, split, grid, st);
    if (r != cudaSuccess || split.kz == 1) return r;
    return launch_pdl(gemm_tc_sum_kernel, dim3((unsigned)((tiles - split.full) * (tn / 8))), dim3(256), 0, st, split, m1, m2, m, tn);
}

// Grouped form over a bank of n_experts Q4_K matrices; slabs of up to `slab` rows (work items of moe_bucket_kernel).
size_t gemm_tc_grouped_record_bytes(int slab, int max_slabs, int in_f) {
    const int n = max_slabs * slab;
    return units_bytes(n, in_f) + extra_bytes(F_Q4, n, in_f);
}
cudaError_t launch_gemm_tc_grouped_prep(int slab, const float *x, void *records, int in_f, const int *slab_expert, const int *slab_p0,
                                        const int *slab_cnt, const int *n_slabs, const int *pair_row, int max_slabs, cudaStream_t st) {
    if (!gemm_tc_takes(DT_Q4K, in_f) || max_slabs < 1 || (uintptr_t)x % 16) return cudaErrorInvalidValue;
    const int n = max_slabs * slab;
    uint8_t *u = static_cast<uint8_t *>(records), *e = u + units_bytes(n, in_f);
    return launch_prep<true>(F_Q4, x, Q8Dev{}, n, slab, in_f, u, e, n, TcGroup{slab_expert, slab_p0, slab_cnt, n_slabs, pair_row}, st);
}
cudaError_t launch_gemm_tc_grouped_silu_prep(int slab, const float *gate, const float *up, void *records, int in_f, const int *slab_expert, const int *slab_p0,
                                             const int *slab_cnt, const int *n_slabs, int max_slabs, cudaStream_t st) {
    if (!gemm_tc_takes(DT_Q4K, in_f) || max_slabs < 1) return cudaErrorInvalidValue;
    const int n = max_slabs * slab;
    uint8_t *u = static_cast<uint8_t *>(records), *e = u + units_bytes(n, in_f);
    return launch_pdl(gemm_tc_silu_prep_kernel<F_Q4>, dim3((unsigned)(((size_t)n * (in_f / 256) + 7) / 8)), dim3(256), 0, st, gate, up, (float *)nullptr, n, slab, in_f, u, e, n,
                      TcGroup{slab_expert, slab_p0, slab_cnt, n_slabs, nullptr});
}
cudaError_t launch_gemm_tc_grouped(int slab, const uint8_t *bank, const uint8_t *bank2, int n_experts, const void *records, float *y, float *y2, int in_f, int out_f,
                                   const int *slab_expert, const int *slab_p0, const int *slab_cnt, const int *n_slabs, int max_slabs,
                                   const DeviceInfo &dev, uint32_t *status, cudaStream_t st) {
    if (!gemm_tc_takes(DT_Q4K, in_f) || out_f < 1 || max_slabs < 1 || n_experts < 1 || (slab != 32 && slab != 64)) return cudaErrorInvalidValue;
    const int n = max_slabs * slab;
    const uint8_t *u = static_cast<const uint8_t *>(records), *e = u + units_bytes(n, in_f);
    CUtensorMap mw, mw2;
    if (!weight_map(F_Q4, bank, (size_t)n_experts * out_f, in_f, &mw) || !weight_map(F_Q4, bank2 ? bank2 : bank, (size_t)n_experts * out_f, in_f, &mw2))
        return cudaErrorInvalidValue;
    TcGroup g{slab_expert, slab_p0, slab_cnt, n_slabs, nullptr};
    TcMat m1{y, out_f}, m2{y2, bank2 ? out_f : 0};
    const int tiles = ((out_f + kTM - 1) / kTM) * (bank2 ? 2 : 1) * max_slabs, cap = ctas_of(F_Q4, slab, dev), grid = tiles < cap ? tiles : cap;
    return launch_tn<F_Q4>(slab, mw, mw2, u, e, m1, m2, n, in_f, status, g, TcSplit{1 << 30, 1, nullptr}, grid, st);
}

}  // namespace infr
