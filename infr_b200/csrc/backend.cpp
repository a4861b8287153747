// CudaBackend: device memory, graph walking and op dispatch (host side).
#include "backend.h"

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>

namespace infr {

namespace {
std::string fmt(const char *f, ...) __attribute__((format(printf, 1, 2)));
std::string fmt(const char *f, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, f);
    vsnprintf(buf, sizeof buf, f, ap);
    va_end(ap);
    return buf;
}
size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
}  // namespace

Status CudaBackend::cuda_status(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return Status::Ok();
    const int32_t code = e == cudaErrorMemoryAllocation ? INFR_E_OOM : INFR_E_CUDA;
    return Status::Err(code, fmt("%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e)));
}

Status CudaBackend::create(const infr_cuda_opts &opts, CudaBackend **out) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n <= 0)
        return Status::Err(INFR_E_CUDA, fmt("no CUDA device: %s (this backend has no CPU fallback)",
                                            e == cudaSuccess ? "device count is 0" : cudaGetErrorString(e)));
    if (opts.device < 0 || opts.device >= n)
        return Status::Err(INFR_E_INVALID, fmt("device %d out of range (%d present)", opts.device, n));
    auto *be = new CudaBackend();
    be->device_ = opts.device;
    be->reference_ = opts.reference != 0;
    Status s;
    if (!(s = be->cuda_status(cudaSetDevice(be->device_), "cudaSetDevice")).ok() ||
        !(s = be->cuda_status(cudaGetDeviceProperties(&be->prop_, be->device_), "cudaGetDeviceProperties")).ok()) {
        delete be;
        return s;
    }
    if (be->prop_.major != 10) {
        s = Status::Err(INFR_E_UNSUPPORTED, fmt("device %d is sm_%d%d; this library is built for sm_100a only",
                                                be->device_, be->prop_.major, be->prop_.minor));
        delete be;
        return s;
    }
    be->dev_.sm_count = be->prop_.multiProcessorCount;
    be->dev_.max_smem_optin = (int)be->prop_.sharedMemPerBlockOptin;
    be->dev_.l2_bytes = (size_t)be->prop_.l2CacheSize;
    if (!(s = be->cuda_status(cudaStreamCreateWithFlags(&be->stream_, cudaStreamNonBlocking), "cudaStreamCreate")).ok() ||
        !(s = be->cuda_status(cudaEventCreate(&be->ev0_), "cudaEventCreate")).ok() ||
        !(s = be->cuda_status(cudaEventCreate(&be->ev1_), "cudaEventCreate")).ok()) {
        delete be;
        return s;
    }
    be->gemv_impl_ = opts.gemv_kernel;
    be->mmq_impl_ = opts.mmq_kernel;
    if (!(s = be->cuda_status(cudaHostAlloc((void **)&be->status_host_, 64, cudaHostAllocMapped), "cudaHostAlloc")).ok() ||
        !(s = be->cuda_status(cudaHostGetDevicePointer((void **)&be->status_dev_, be->status_host_, 0), "cudaHostGetDevicePointer")).ok()) {
        delete be;
        return s;
    }
    *be->status_host_ = 0;
    if (!(s = be->cuda_status(cudaHostAlloc((void **)&be->up_ring_, kUpSlots * kUpSlotBytes, cudaHostAllocDefault), "cudaHostAlloc(upload ring)")).ok()) {
        delete be;
        return s;
    }
    for (int i = 0; i < kUpSlots; i++)
        if (!(s = be->cuda_status(cudaEventCreateWithFlags(&be->up_ev_[i], cudaEventDisableTiming), "cudaEventCreate")).ok()) {
            delete be;
            return s;
        }
    *out = be;
    return Status::Ok();
}

// A kernel whose bounded wait expired leaves a non-zero word in mapped host memory.
Status CudaBackend::check_device_status() {
    if (status_host_ && *(volatile uint32_t *)status_host_) {
        const uint32_t v = *(volatile uint32_t *)status_host_;
        *(volatile uint32_t *)status_host_ = 0;
        return Status::Err(INFR_E_TIMEOUT, fmt("a device-side wait expired (kernel status %u); results of this stream are invalid", v));
    }
    return Status::Ok();
}

CudaBackend::~CudaBackend() {
    cudaSetDevice(device_);
    if (stream_) cudaStreamSynchronize(stream_);
    if (scratch_) cudaFree(scratch_);
    if (flush_) cudaFree(flush_);
    for (auto &b : pool_) cudaFree(b.ptr);
    if (status_host_) cudaFreeHost(status_host_);
    if (up_ring_) cudaFreeHost(up_ring_);
    for (cudaEvent_t e : up_ev_)
        if (e) cudaEventDestroy(e);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    if (stream_) cudaStreamDestroy(stream_);
}

infr_cuda_caps CudaBackend::capabilities() const {
    infr_cuda_caps c;
    memset(&c, 0, sizeof c);
    snprintf(c.name, sizeof c.name, "%s", name());
    c.f16 = 1;
    c.i8 = 1;
    c.i8_dot = 1;
    c.integrated = 0;
    c.unified_memory = 0;
    c.decode_replay = 0;
    c.graph_input_inplace = 1;
    c.max_shared_memory_bytes = (uint32_t)dev_.max_smem_optin;
    c.sm_count = (uint32_t)dev_.sm_count;
    c.total_memory_bytes = (uint64_t)prop_.totalGlobalMem;
    c.l2_bytes = (uint64_t)dev_.l2_bytes;
    return c;
}

// ---------------------------------------------------------------------------------------- memory
Status CudaBackend::alloc(size_t bytes, int usage, bool zero, infr_cuda_buf **out) {
    if (capturing_) return Status::Err(INFR_E_INVALID, "alloc during stream capture");
    cudaSetDevice(device_);
    void *p = nullptr;
    // Round up so 16-byte vector accesses on the tail of a row never leave the allocation.
    const size_t padded = align_up(bytes ? bytes : 1, 256);
    Status s = cuda_status(cudaMalloc(&p, padded), "cudaMalloc");
    if (!s.ok()) return s;
    if (zero) {
        s = cuda_status(cudaMemsetAsync(p, 0, padded, stream_), "cudaMemsetAsync");
    } else {
        // only the padding must be defined
        if (padded > bytes) s = cuda_status(cudaMemsetAsync((uint8_t *)p + bytes, 0, padded - bytes, stream_), "cudaMemsetAsync");
    }
    if (!s.ok()) {
        cudaFree(p);
        return s;
    }
    auto *b = new infr_cuda_buf();
    b->ptr = p;
    b->len = bytes;
    b->usage = usage;
    b->uid = next_uid_++;
    *out = b;
    return Status::Ok();
}

Status CudaBackend::wrap(void *device_ptr, size_t bytes, int usage, infr_cuda_buf **out) {
    if (!device_ptr || !bytes) return Status::Err(INFR_E_INVALID, "wrap: null pointer or empty range");
    if ((uintptr_t)device_ptr % 16) return Status::Err(INFR_E_INVALID, "wrap: the device pointer must be 16-byte aligned");
    auto *b = new infr_cuda_buf();
    b->ptr = device_ptr;
    b->len = bytes;
    b->usage = usage;
    b->uid = next_uid_++;
    b->owned = false;
    *out = b;
    return Status::Ok();
}

void CudaBackend::free_buffer(infr_cuda_buf *b) {
    if (!b) return;
    cudaSetDevice(device_);
    if (!capturing_ && b->owned) cudaStreamSynchronize(stream_);  // a non-owning handle frees nothing
    if (b->owned) cudaFree(b->ptr);
    delete b;
}

Status CudaBackend::upload(infr_cuda_buf *dst, size_t dst_off, const void *src, size_t bytes) {
    if (!dst || (!src && bytes)) return Status::Err(INFR_E_INVALID, "upload: null argument");
    if (dst_off > dst->len || bytes > dst->len - dst_off)
        return Status::Err(INFR_E_INVALID, fmt("upload: %zu bytes at offset %zu into a %zu-byte buffer", bytes, dst_off, dst->len));
    if (capturing_) return Status::Err(INFR_E_INVALID, "upload during stream capture");
    cudaSetDevice(device_);
    // The caller may reuse `src` as soon as this returns (the trait takes a borrowed slice).  A small upload (a
    // decode step's activations) is copied into a pinned slot of the context's ring and sent from there, so that
    // the call returns without waiting for the stream; a slot is reused only after its copy has completed.
    if (bytes <= kUpSlotBytes) {
        const int slot = up_next_;
        up_next_ = (up_next_ + 1) % kUpSlots;
        Status s = cuda_status(cudaEventSynchronize(up_ev_[slot]), "upload slot");
        if (!s.ok()) return s;
        uint8_t *stage = up_ring_ + (size_t)slot * kUpSlotBytes;
        memcpy(stage, src, bytes);
        s = cuda_status(cudaMemcpyAsync((uint8_t *)dst->ptr + dst_off, stage, bytes, cudaMemcpyHostToDevice, stream_), "upload");
        if (!s.ok()) return s;
        return cuda_status(cudaEventRecord(up_ev_[slot], stream_), "upload event");
    }
    Status s = cuda_status(cudaMemcpyAsync((uint8_t *)dst->ptr + dst_off, src, bytes, cudaMemcpyHostToDevice, stream_), "upload");
    if (!s.ok()) return s;
    return cuda_status(cudaStreamSynchronize(stream_), "upload sync");
}

Status CudaBackend::download(const infr_cuda_buf *src, void *dst, size_t bytes) {
    if (!src || (!dst && bytes)) return Status::Err(INFR_E_INVALID, "download: null argument");
    if (bytes > src->len)
        return Status::Err(INFR_E_INVALID, fmt("download: %zu bytes from a %zu-byte buffer", bytes, src->len));
    if (capturing_) return Status::Err(INFR_E_INVALID, "download during stream capture");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaMemcpyAsync(dst, src->ptr, bytes, cudaMemcpyDeviceToHost, stream_), "download");
    if (!s.ok()) return s;
    s = cuda_status(cudaStreamSynchronize(stream_), "download sync");
    return s.ok() ? check_device_status() : s;
}

Status CudaBackend::copy_buffer(const infr_cuda_buf *src, infr_cuda_buf *dst, size_t bytes) {
    if (!src || !dst) return Status::Err(INFR_E_INVALID, "copy: null buffer");
    if (bytes > src->len || bytes > dst->len)
        return Status::Err(INFR_E_INVALID, fmt("copy: %zu bytes between %zu- and %zu-byte buffers", bytes, src->len, dst->len));
    cudaSetDevice(device_);
    return cuda_status(cudaMemcpyAsync(dst->ptr, src->ptr, bytes, cudaMemcpyDeviceToDevice, stream_), "copy");
}

Status CudaBackend::sync() {
    if (capturing_) return Status::Err(INFR_E_INVALID, "sync during stream capture");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaStreamSynchronize(stream_), "sync");
    return s.ok() ? check_device_status() : s;
}

Status CudaBackend::ensure_scratch(size_t bytes) {
    if (bytes <= scratch_bytes_) return Status::Ok();
    if (capturing_)
        return Status::Err(INFR_E_INVALID, "activation scratch would grow during stream capture; run the same calls once before capturing");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaStreamSynchronize(stream_), "scratch sync");
    if (!s.ok()) return s;
    if (scratch_) cudaFree(scratch_);
    scratch_ = nullptr;
    scratch_bytes_ = 0;
    const size_t want = align_up(bytes, 1 << 20);
    s = cuda_status(cudaMalloc(&scratch_, want), "scratch cudaMalloc");
    if (!s.ok()) return s;
    scratch_bytes_ = want;
    scratch_gen_++;
    return Status::Ok();
}

// ------------------------------------------------------------------------------------------- ops
Status CudaBackend::quantize_q8(int gran, const float *x, uint32_t rows, uint32_t k, int8_t *qs, float *d,
                                int32_t *sums, int32_t *sums16, uint16_t *dact, uint16_t *sact) {
    if (gran != 32 && gran != 256) return Status::Err(INFR_E_INVALID, fmt("quantize_q8: granularity %d (32 or 256)", gran));
    if (k == 0 || k % (uint32_t)gran) return Status::Err(INFR_E_INVALID, fmt("quantize_q8: k=%u is not a multiple of %d", k, gran));
    cudaSetDevice(device_);
    Status s = cuda_status(launch_quantize_q8(x, (int)rows, (int)k, gran, qs, d, sums, sums16, dact, sact, stream_), "quantize_q8");
    if (s.ok() && rows) launches_++;
    return s;
}

// Lays the quantised rows out in the context scratch: qs | d | sums | sums16.
Status CudaBackend::quantize_for(int dtype, const float *x, uint32_t rows, uint32_t k, Q8Dev *out, size_t extra, uint8_t **extra_ptr) {
    const int gran = act_gran(dtype);
    const size_t qs_b = align_up((size_t)rows * k, 256);
    const size_t d_b = align_up((size_t)rows * (k / gran) * 4, 256);
    const size_t s_b = align_up((size_t)rows * (k / 32) * 4, 256);
    const size_t s16_b = dtype == DT_Q6K ? align_up((size_t)rows * (k / 16) * 4, 256) : 0;
    Status s = ensure_scratch(qs_b + d_b + s_b + s16_b + align_up(extra, 256));
    if (!s.ok()) return s;
    uint8_t *p = scratch();
    if (extra_ptr) *extra_ptr = p + qs_b + d_b + s_b + s16_b;
    int8_t *qs = reinterpret_cast<int8_t *>(p);
    float *d = reinterpret_cast<float *>(p + qs_b);
    int32_t *sums = reinterpret_cast<int32_t *>(p + qs_b + d_b);
    int32_t *sums16 = s16_b ? reinterpret_cast<int32_t *>(p + qs_b + d_b + s_b) : nullptr;
    s = quantize_q8(gran, x, rows, k, qs, d, sums, sums16, nullptr, nullptr);
    if (!s.ok()) return s;
    *out = Q8Dev{qs, d, sums, sums16, gran};
    return Status::Ok();
}

// Up to 8 quantised rows through the GEMV of the format; rows so long that m of them staged exceed shared memory in narrower batches.
Status CudaBackend::gemv_q8_rows(int dtype, const uint8_t *w, const Q8Dev &a, float *y, uint32_t m, uint32_t in_f, uint32_t out_f) {
    uint32_t step = m;
    for (uint32_t t0 = 0; t0 < m;) {
        const uint32_t n = m - t0 < step ? m - t0 : step;
        Q8Dev sub = a;
        sub.qs = a.qs + (size_t)t0 * in_f;
        sub.d = a.d + (size_t)t0 * (in_f / a.gran);
        sub.sums = a.sums + (size_t)t0 * (in_f / 32);
        if (a.sums16) sub.sums16 = a.sums16 + (size_t)t0 * (in_f / 16);
        float *yt = y + (size_t)t0 * out_f;
        const cudaError_t e = gemv_impl_ == 1   ? launch_gemv_q8(dtype, w, sub, yt, (int)n, (int)in_f, (int)out_f, nullptr, dev_, stream_)
                              : dtype == DT_Q4K ? launch_gemv_q4k_mma(w, &sub, nullptr, yt, (int)n, (int)in_f, (int)out_f, dev_, status_dev_, stream_)
                                                : launch_gemv_stream(dtype, w, sub, yt, (int)n, (int)in_f, (int)out_f, dev_, status_dev_, stream_);
        if (e == cudaErrorInvalidValue && step > 1) {
            cudaGetLastError();
            step /= 2;
            continue;
        }
        Status s = cuda_status(e, "gemv_q8");
        if (!s.ok()) return s;
        launches_ += 1;
        t0 += n;
    }
    return Status::Ok();
}

static bool overlap(const float *a, size_t na, const float *b, size_t nb) {
    return (uintptr_t)a < (uintptr_t)b + nb * 4 && (uintptr_t)b < (uintptr_t)a + na * 4;
}

Status CudaBackend::linear(int dtype, const uint8_t *w, const float *x, float *y, uint32_t m, uint32_t in_f,
                           uint32_t out_f, int act) {
    if (dtype != DT_Q4K && dtype != DT_Q6K && dtype != DT_Q2_0)
        return Status::Err(INFR_E_UNSUPPORTED, fmt("linear: weight dtype code %d is not supported (Q4_K, Q6_K, Q2_0)", dtype));
    if (act != INFR_ACT_INT8 && act != INFR_ACT_F32) return Status::Err(INFR_E_INVALID, fmt("linear: activation mode %d", act));
    const int be = block_elems(dtype);
    if (in_f == 0 || in_f % (uint32_t)be) return Status::Err(INFR_E_INVALID, fmt("linear: in_f=%u is not a whole number of %d-element blocks", in_f, be));
    if (in_f % 16) return Status::Err(INFR_E_INVALID, fmt("linear: in_f=%u must be a multiple of 16", in_f));
    if (m == 0 || out_f == 0) return Status::Ok();
    cudaSetDevice(device_);
    // More than 8 rows with int8 activations.  Q4_K and Q6_K: up to 32 rows (a decode step over that many sequences) take
    // the wide GEMV, more the tensor-memory GEMM (gemv_rows has the measured lines; rows that the GEMM's tiled copies cannot fetch
    // are walked).  Q2_0: the batched GEMM on the warp matrix unit.  mmq_kernel 1: the bit-identical GEMM for
    // Q4_K, 2: the tensor-memory GEMM for every batch above 8 rows, 3: everything through the GEMV 8 rows at a time (the
    // parity tests and the bench compare them).
    if (wide_applies(dtype, m, in_f, out_f, act) && !tc_wins(dtype, m, in_f, out_f)) {
        Q8Dev a;
        uint8_t *partials = nullptr;
        Status s = quantize_for(dtype, x, m, in_f, &a, gemv_wide_partial_bytes(m < 32 ? (int)m : 32, (int)in_f, (int)out_f), &partials);
        return s.ok() ? wide_gemm(dtype, w, a, y, m, in_f, out_f, reinterpret_cast<float *>(partials)) : s;
    }
    if (m > 8 && dtype == DT_Q4K && act == INFR_ACT_INT8 && gemv_impl_ == 0 && mmq_impl_ == 1) {
        Q8Dev a;
        uint8_t *rec = nullptr;
        Status s = quantize_for(dtype, x, m, in_f, &a, mmq_q4k_record_bytes((int)m, (int)in_f), &rec);
        if (!s.ok()) return s;
        s = cuda_status(launch_mmq_q4k(w, a, rec, y, (int)m, (int)in_f, (int)out_f, dev_, status_dev_, stream_), "mmq_q4k");
        if (s.ok()) launches_ += 2;
        return s;
    }
    if (q2_applies(dtype, m, in_f, act)) return q2_linear(w, y, out_f, nullptr, nullptr, 0, x, m, in_f);
    if (tc_applies(dtype, m, in_f, out_f, act) || (wide_applies(dtype, m, in_f, out_f, act) && tc_wins(dtype, m, in_f, out_f)))
        return tc_linear(dtype, w, y, out_f, nullptr, nullptr, 0, x, nullptr, m, in_f);
    // Kernels that read the f32 rows in every CTA need a result apart from them: in place the rows are quantised first.
    const bool in_place = overlap(x, (size_t)m * in_f, y, (size_t)m * out_f);
    // One Q2_0 row: quantised inside the GEMV, unless it is so long that every CTA's own quantising costs more than a launch.  Quantiser and
    // GEMV / one launch (us, cold weights): 8192 -> 8192 8.5 / 9.2, 14336 -> 4096 9.6 / 9.5, -> 8192 12.6 / 14.6, 16384 -> 4096 10.2 / 9.8,
    // 20480 -> 4096 13.0 / 12.6, 53248 -> 4096 24 / 32, 65536 -> 2048 19 / 21.  (A pair saves two launches: always.)
    if (dtype == DT_Q2_0 && m == 1 && (in_f <= 4096 || (in_f <= 28672 && out_f <= 32u * (uint32_t)dev_.sm_count)) && act == INFR_ACT_INT8 && gemv_impl_ == 0 && !in_place) {
        const cudaError_t e = launch_gemv_q2_row(w, y, (int)out_f, nullptr, nullptr, 0, x, (int)in_f, dev_, status_dev_, stream_);
        if (e == cudaSuccess) launches_++;
        if (e != cudaErrorInvalidValue) return cuda_status(e, "gemv_q2");
        cudaGetLastError();
    }
    // One Q6_K row: the same (16384 -> 4096 15.4 / 14.6, 20480 -> 4096 18.1 / 18.0, 24576 -> 2048 13.7 / 14.1, 32768 -> 2048 17 / 19).
    if (dtype == DT_Q6K && m == 1 && in_f <= 20480 && act == INFR_ACT_INT8 && gemv_impl_ == 0 && !in_place && gemv_row_takes(dtype, (int)in_f)) {
        const GemvRowMat mat{w, y, (int)out_f};
        const cudaError_t e = launch_gemv_row(GemvRow{dtype, (int)in_f, &mat, 1, nullptr, x}, dev_, status_dev_, stream_);
        if (e == cudaSuccess) launches_++;
        if (e != cudaErrorInvalidValue) return cuda_status(e, "gemv_row");
        cudaGetLastError();
    }
    if (act == INFR_ACT_F32 && in_place) {  // the f32 kernels read the rows while they store: from a copy
        Status s = ensure_scratch((size_t)m * in_f * 4);
        if (s.ok()) s = cuda_status(cudaMemcpyAsync(scratch(), x, (size_t)m * in_f * 4, cudaMemcpyDeviceToDevice, stream_), "linear: rows");
        if (!s.ok()) return s;
        x = reinterpret_cast<const float *>(scratch());
    }
    // Decode shapes (m <= 8) run the streaming GEMV; wider batches are walked 8 rows at a time, all rows quantised once.
    Q8Dev a_all{};
    // (a single Q4_K chunk quantises its rows inside the GEMV; with several chunks that would repeat the work in every CTA)
    const bool pre_quantised = act == INFR_ACT_INT8 && (!(dtype == DT_Q4K && gemv_impl_ == 0) || m > 8 || in_place);
    if (pre_quantised) {
        Status s = quantize_for(dtype, x, m, in_f, &a_all);
        if (!s.ok()) return s;
    }
    for (uint32_t r0 = 0; r0 < m; r0 += 8) {
        const uint32_t mm = m - r0 < 8 ? m - r0 : 8;
        const float *xr = x + (size_t)r0 * in_f;
        float *yr = y + (size_t)r0 * out_f;
        if (act == INFR_ACT_F32) {
            Status s = cuda_status(launch_gemv_f32(dtype, w, xr, yr, (int)mm, (int)in_f, (int)out_f, dev_, stream_), "gemv_f32");
            if (!s.ok()) return s;
            launches_ += 1;
        } else if (!pre_quantised) {
            // Q4_K, one kernel: activation rows are quantised inside the GEMV while the first weights stream in.
            // Rows so long that `mm` staged activation rows exceed shared memory are run in narrower batches.
            uint32_t step = mm;
            for (uint32_t t0 = 0; t0 < mm;) {
                const uint32_t n = mm - t0 < step ? mm - t0 : step;
                cudaError_t e = launch_gemv_q4k_mma(w, nullptr, xr + (size_t)t0 * in_f, yr + (size_t)t0 * out_f, (int)n, (int)in_f,
                                                    (int)out_f, dev_, status_dev_, stream_);
                if (e == cudaErrorInvalidValue && step > 1) {
                    cudaGetLastError();
                    step /= 2;
                    continue;
                }
                Status s = cuda_status(e, "gemv_q4k");
                if (!s.ok()) return s;
                launches_ += 1;
                t0 += n;
            }
        } else {
            // this chunk's rows of the quantised batch
            Q8Dev a = a_all;
            a.qs = a_all.qs + (size_t)r0 * in_f;
            a.d = a_all.d + (size_t)r0 * (in_f / a.gran);
            a.sums = a_all.sums + (size_t)r0 * (in_f / 32);
            if (a_all.sums16) a.sums16 = a_all.sums16 + (size_t)r0 * (in_f / 16);
            Status s = gemv_q8_rows(dtype, w, a, yr, mm, in_f, out_f);
            if (!s.ok()) return s;
        }
    }
    return Status::Ok();
}

// Rows up to which a batch takes the wide GEMV where the GEMM could run too; out_f: the height of all weights of the call.
// Measured, GEMV / GEMM (us): Q4_K 32 rows 4096 -> 14336 27 / 26, 4096 -> 4096 13 / 17.  Q6_K 32 rows 4096 -> 14336 33 / 41, 33 rows
// 54 / 41; against few weights a second pass costs less than the GEMM's two other launches: 2048 -> 2048 33 rows 12.1 / 13.6, 48 rows
// 13.9 / 15.7, 4096 -> 1024 33 rows 15.0 / 16.1, but 4096 -> 512 15.4 / 13.4 and 4096 -> 2048 18.8 / 17.7.
static uint32_t gemv_rows(int dtype, uint32_t in_f, uint64_t out_f) {
    return dtype == DT_Q6K && 4 * out_f >= in_f && out_f * in_f <= (4u << 20) ? 48 : 32;
}

bool CudaBackend::wide_applies(int dtype, uint32_t m, uint32_t in_f, uint64_t out_f, int act) const {
    if (act != INFR_ACT_INT8 || m <= 8 || gemv_impl_ != 0 || mmq_impl_ != 0 || in_f == 0 || in_f % 256) return false;
    if (m > gemv_rows(dtype, in_f, out_f)) return false;
    if (dtype == DT_Q4K) return true;
    if (dtype == DT_Q6K) return in_f % 2048 == 0;  // (rows of a whole number of 16-byte units: the TMA stride rule)
    return false;
}

// y[m, out_f] from quantised rows, 32 rows per pass of the weights.
// w2 / y2 / out_f2: a second weight against the same rows in the same launches (partials sized for out_f + out_f2).
Status CudaBackend::wide_gemm(int dtype, const uint8_t *w, const Q8Dev &a, float *y, uint32_t m, uint32_t in_f, uint32_t out_f, float *partials,
                              const uint8_t *w2, float *y2, uint32_t out_f2) {
    const uint32_t nb = in_f / 256;
    for (uint32_t r0 = 0; r0 < m; r0 += 32) {
        const uint32_t mm = m - r0 < 32 ? m - r0 : 32;
        Q8Dev sub = a;
        sub.qs = a.qs + (size_t)r0 * in_f;
        sub.d = a.d + (size_t)r0 * nb;
        sub.sums = a.sums + (size_t)r0 * nb * 8;
        if (a.sums16) sub.sums16 = a.sums16 + (size_t)r0 * nb * 16;
        Status s = cuda_status(launch_gemv_wide(dtype, w, sub, y + (size_t)r0 * out_f, partials, (int)mm, (int)in_f, (int)out_f, dev_, status_dev_, stream_,
                                                nullptr, w2, y2 ? y2 + (size_t)r0 * out_f2 : nullptr, (int)out_f2),
                               "gemv_wide");
        if (!s.ok()) return s;
        launches_ += (uint64_t)gemv_wide_launches((int)in_f);
    }
    return Status::Ok();
}

bool CudaBackend::tc_applies(int dtype, uint32_t m, uint32_t in_f, uint64_t out_f, int act) const {
    if (act != INFR_ACT_INT8 || m <= 8 || gemv_impl_ != 0 || (mmq_impl_ != 0 && mmq_impl_ != 2) || !gemm_tc_takes(dtype, (int)in_f)) return false;
    return mmq_impl_ == 2 || m > gemv_rows(dtype, in_f, out_f);
}

// Where the wide GEMV applies too: a batch against enough Q4_K weights that the GEMM's fixed cost (the layout launch and the
// pipeline's start) is paid back and so many rows that the wide GEMV multiplies four groups of eight.  Measured, wide GEMV /
// GEMM (us): 4096 -> 2 x 14336 at 16 rows 32 / 37, 24 rows 38 / 37, 32 rows 47 / 37; 4096 -> 2 x 8192 at 24 rows 25 / 25, 32 rows
// 30 / 26; 2048 -> 2 x 8192 at 32 rows 18.4 / 17.7; 4096 -> 4096 + 1024 at 32 rows 15 / 18.
bool CudaBackend::tc_wins(int dtype, uint32_t m, uint32_t in_f, uint64_t out_f) const {
    if (dtype != DT_Q4K || !gemm_tc_takes(dtype, (int)in_f)) return false;
    return m > 24 && out_f * in_f >= (48u << 20);
}

size_t CudaBackend::tc_scratch_bytes(int dtype, uint32_t m, uint32_t in_f, uint32_t out_f1, uint32_t out_f2) const {
    return align_up(gemm_tc_record_bytes(dtype, (int)m, (int)in_f), 256) +
           align_up(gemm_tc_partial_bytes(dtype, (int)m, (int)in_f, (int)out_f1, (int)out_f2, dev_), 256);
}

// One weight, or two against the same rows in one launch.  The context scratch holds the operand layout of the rows and the
// K-split partial results behind it.
Status CudaBackend::tc_linear(int dtype, const uint8_t *w, float *y, uint32_t out_f, const uint8_t *w2, float *y2, uint32_t out_f2, const float *x,
                              const Q8Dev *a, uint32_t m, uint32_t in_f, const RowSource *src) {
    const size_t rec = align_up(gemm_tc_record_bytes(dtype, (int)m, (int)in_f), 256);
    const size_t part = gemm_tc_partial_bytes(dtype, (int)m, (int)in_f, (int)out_f, (int)out_f2, dev_);
    Status s = ensure_scratch(tc_scratch_bytes(dtype, m, in_f, out_f, out_f2));
    if (!s.ok()) return s;
    s = cuda_status(src ? launch_gemm_tc_prep(dtype, *src, scratch(), (int)m, (int)in_f, stream_) : launch_gemm_tc_prep(dtype, x, a, scratch(), (int)m, (int)in_f, stream_),
                    "gemm_tc layout");
    if (!s.ok()) return s;
    s = cuda_status(launch_gemm_tc(dtype, w, scratch(), y, part ? reinterpret_cast<float *>(scratch() + rec) : nullptr, (int)m, (int)in_f, (int)out_f, dev_,
                                   status_dev_, stream_, w2, y2, (int)out_f2),
                    "gemm_tc");
    if (s.ok()) launches_ += 2 + (part ? 1 : 0);
    return s;
}

// Q2_0, more than 8 rows: the batched GEMM on the warp matrix unit (mmq_kernel 3 walks them 8 at a time).
bool CudaBackend::q2_applies(int dtype, uint32_t m, uint32_t in_f, int act) const {
    return dtype == DT_Q2_0 && m > 8 && act == INFR_ACT_INT8 && gemv_impl_ == 0 && (mmq_impl_ == 0 || mmq_impl_ == 2) && gemm_q2_takes((int)in_f);
}

// One weight, or two against the same rows in one launch; the context scratch holds the laid-out rows and the K-split parts.
Status CudaBackend::q2_linear(const uint8_t *w, float *y, uint32_t out_f, const uint8_t *w2, float *y2, uint32_t out_f2, const float *x, uint32_t m,
                              uint32_t in_f) {
    const size_t rec = gemm_q2_record_bytes((int)m, (int)in_f), part = gemm_q2_partial_bytes((int)m, (int)in_f, (int)out_f, (int)out_f2, dev_);
    Status s = ensure_scratch(rec + part);
    if (!s.ok()) return s;
    s = cuda_status(launch_gemm_q2_prep(x, scratch(), (int)m, (int)in_f, stream_), "gemm_q2 layout");
    if (!s.ok()) return s;
    s = cuda_status(launch_gemm_q2(w, scratch(), y, part ? reinterpret_cast<float *>(scratch() + rec) : nullptr, (int)m, (int)in_f, (int)out_f, dev_,
                                   status_dev_, stream_, w2, y2, (int)out_f2),
                    "gemm_q2");
    if (s.ok()) launches_ += 2 + (part ? 1 : 0);
    return s;
}

bool CudaBackend::tc_rows(int dtype, uint32_t m, uint32_t in_f, uint64_t out_f) const {
    if (reference_ || (dtype != DT_Q4K && dtype != DT_Q6K) || m == 0 || out_f == 0) return false;
    const bool wide = wide_applies(dtype, m, in_f, out_f, INFR_ACT_INT8);
    return wide ? tc_wins(dtype, m, in_f, out_f) : tc_applies(dtype, m, in_f, out_f, INFR_ACT_INT8);
}

Status CudaBackend::linear_from(const RowSource &src, int dtype, const uint8_t *w1, float *y1, uint32_t out_f1, const uint8_t *w2, float *y2, uint32_t out_f2, uint32_t m,
                                uint32_t in_f, bool *taken) {
    *taken = false;
    const size_t n = (size_t)m * in_f;
    if (!tc_rows(dtype, m, in_f, (uint64_t)out_f1 + out_f2) || !out_f1 || (w2 && !out_f2)) return Status::Ok();
    if (((uintptr_t)src.a | (uintptr_t)src.b | (uintptr_t)src.sum | (uintptr_t)src.norm_w | (uintptr_t)src.dst) % 16) return Status::Ok();
    auto apart = [&](const float *p) { return !p || p == src.dst || !overlap(p, n, src.dst, n); };
    if (!apart(src.a) || !apart(src.b) || !apart(src.sum)) return Status::Ok();
    *taken = true;
    cudaSetDevice(device_);
    return tc_linear(dtype, w1, y1, out_f1, w2, y2, out_f2, nullptr, nullptr, m, in_f, &src);
}

// Two weights of one format against the same f32 rows (q and k, gate and up): the rows are quantised once.
Status CudaBackend::linear_pair(int dtype, const uint8_t *w1, float *y1, uint32_t out_f1, const uint8_t *w2, float *y2, uint32_t out_f2,
                                const float *x, uint32_t m, uint32_t in_f, int act) {
    const uint64_t both = (uint64_t)out_f1 + out_f2;
    const bool wide = wide_applies(dtype, m, in_f, both, act), gemm = wide && tc_wins(dtype, m, in_f, both);
    if (wide && !gemm && out_f1 && out_f2) {
        cudaSetDevice(device_);
        const int mm = m < 32 ? (int)m : 32;
        Q8Dev a;
        uint8_t *partials = nullptr;
        Status s = quantize_for(dtype, x, m, in_f, &a, gemv_wide_partial_bytes(mm, (int)in_f, (int)(out_f1 + out_f2)), &partials);
        return s.ok() ? wide_gemm(dtype, w1, a, y1, m, in_f, out_f1, reinterpret_cast<float *>(partials), w2, y2, out_f2) : s;
    }
    if (q2_applies(dtype, m, in_f, act) && out_f1 && out_f2) {
        cudaSetDevice(device_);
        return q2_linear(w1, y1, out_f1, w2, y2, out_f2, x, m, in_f);
    }
    if ((gemm || tc_applies(dtype, m, in_f, both, act)) && out_f1 && out_f2) {
        cudaSetDevice(device_);
        return tc_linear(dtype, w1, y1, out_f1, w2, y2, out_f2, x, nullptr, m, in_f);
    }
    if (act == INFR_ACT_INT8 && m >= 1 && m <= 8 && (dtype == DT_Q4K || dtype == DT_Q6K || dtype == DT_Q2_0) && in_f &&
        in_f % (uint32_t)block_elems(dtype) == 0 && in_f % 16 == 0 && out_f1 && out_f2) {
        cudaSetDevice(device_);
        // (in place: quantise first; results that overlap each other: one launch each, in order)
        const size_t nx = (size_t)m * in_f, n1 = (size_t)m * out_f1, n2 = (size_t)m * out_f2;
        const bool apart = !overlap(x, nx, y1, n1) && !overlap(x, nx, y2, n2) && !overlap(y1, n1, y2, n2);
        if (m == 1 && gemv_impl_ == 0 && apart && dtype == DT_Q6K && in_f <= 36864 && gemv_row_takes(dtype, (int)in_f)) {
            const GemvRowMat mats[2] = {{w1, y1, (int)out_f1, nullptr, (int)out_f2}, {w2, y2, (int)out_f2, nullptr, (int)out_f1}};
            const cudaError_t e = launch_gemv_row(GemvRow{dtype, (int)in_f, mats, 2, nullptr, x}, dev_, status_dev_, stream_);
            if (e == cudaSuccess) launches_++;
            if (e != cudaErrorInvalidValue) return cuda_status(e, "linear_pair");
            cudaGetLastError();
        }
        if (dtype == DT_Q4K && gemv_impl_ == 0 && in_f % 256 == 0 && apart) {
            // one kernel: the rows are quantised inside the GEMV while the first weights stream in
            const cudaError_t e = launch_gemv_q4k_mma_pair(w1, y1, (int)out_f1, w2, y2, (int)out_f2, nullptr, x, (int)m, (int)in_f, dev_,
                                                           status_dev_, stream_);
            if (e == cudaSuccess) {
                launches_++;
                return Status::Ok();
            }
            if (e != cudaErrorInvalidValue) return cuda_status(e, "linear_pair");
            cudaGetLastError();  // rows too long to stage m of them in one CTA: quantise first
        }
        if (dtype == DT_Q2_0 && m == 1 && gemv_impl_ == 0 && apart) {
            const cudaError_t e = launch_gemv_q2_row(w1, y1, (int)out_f1, w2, y2, (int)out_f2, x, (int)in_f, dev_, status_dev_, stream_);
            if (e == cudaSuccess) launches_++;
            if (e != cudaErrorInvalidValue) return cuda_status(e, "linear_pair");
            cudaGetLastError();  // a row too long to stage: quantise first
        }
        Q8Dev a;
        Status s = quantize_for(dtype, x, m, in_f, &a);
        if (s.ok()) s = gemv_q8_rows(dtype, w1, a, y1, m, in_f, out_f1);
        return s.ok() ? gemv_q8_rows(dtype, w2, a, y2, m, in_f, out_f2) : s;
    }
    Status s = linear(dtype, w1, x, y1, m, in_f, out_f1, act);
    return s.ok() ? linear(dtype, w2, x, y2, m, in_f, out_f2, act) : s;
}

Status CudaBackend::linear_row(const GemvRow &d, bool *taken) {
    *taken = false;
    if (reference_ || gemv_impl_ != 0 || !gemv_row_takes(d.dtype, d.in_f) || d.n < 1 || d.n > kGemvRowMats) return Status::Ok();
    // Every CTA reads its row while others store: results lie apart from what is read and from each other.
    struct Span {
        uintptr_t a, b;
        bool w;
    } sp[2 * kGemvRowMats + 1];
    int n = 0;
    auto put = [&](const float *p, size_t k, bool w) {
        if (p) sp[n++] = Span{(uintptr_t)p, (uintptr_t)p + 4 * k, w};
    };
    put(d.x, (size_t)d.in_f, false);
    for (int i = 0; i < d.n; i++) {
        put(d.mats[i].x, (size_t)d.in_f, false);
        put(d.mats[i].y, (size_t)d.mats[i].out_f, true);
    }
    std::sort(sp, sp + n, [](const Span &p, const Span &q) { return p.a < q.a; });
    uintptr_t end_any = 0, end_written = 0;
    for (int i = 0; i < n; i++) {
        if (sp[i].a < (sp[i].w ? end_any : end_written)) return Status::Ok();
        if (sp[i].b > end_any) end_any = sp[i].b;
        if (sp[i].w && sp[i].b > end_written) end_written = sp[i].b;
    }
    cudaSetDevice(device_);
    const cudaError_t e = launch_gemv_row(d, dev_, status_dev_, stream_);
    if (e == cudaErrorInvalidValue) {
        cudaGetLastError();
        return Status::Ok();
    }
    Status s = cuda_status(e, "gemv_row");
    if (s.ok()) launches_++;
    *taken = true;
    return s;
}

Status CudaBackend::gemv_q8(int dtype, const uint8_t *w, const Q8Dev &a, float *y, uint32_t m, uint32_t in_f, uint32_t out_f) {
    if (dtype != DT_Q4K && dtype != DT_Q6K && dtype != DT_Q2_0)
        return Status::Err(INFR_E_UNSUPPORTED, fmt("gemv_q8: weight dtype code %d", dtype));
    const bool wide = m > 8 && wide_applies(dtype, m, in_f, out_f, INFR_ACT_INT8);
    // (Q6_K rows above what the wide GEMV takes: the tensor-memory GEMM)
    const bool tc = dtype == DT_Q6K && mmq_impl_ == 0 && tc_applies(dtype, m, in_f, out_f, INFR_ACT_INT8);
    if (m == 0 || (m > 8 && !wide && !tc))
        return Status::Err(INFR_E_INVALID, fmt("gemv_q8: m=%u (1..8; more rows where the wide GEMV applies: Q4_K up to 32, Q6_K with in_f a multiple of 2048)", m));
    if (in_f == 0 || in_f % (uint32_t)block_elems(dtype) || in_f % 16) return Status::Err(INFR_E_INVALID, fmt("gemv_q8: in_f=%u", in_f));
    if (a.gran != act_gran(dtype)) return Status::Err(INFR_E_INVALID, fmt("gemv_q8: activations have granularity %d, dtype needs %d", a.gran, act_gran(dtype)));
    if (dtype == DT_Q6K && !a.sums16) return Status::Err(INFR_E_INVALID, "gemv_q8: Q6_K needs the per-16 sums");
    cudaSetDevice(device_);
    if (tc || (wide && tc_wins(dtype, m, in_f, out_f))) return tc_linear(dtype, w, y, out_f, nullptr, nullptr, 0, nullptr, &a, m, in_f);
    if (wide) {
        // a decode batch of a few dozen rows: the context scratch holds the partial results of the K chunks
        const size_t pb = gemv_wide_partial_bytes(m < 32 ? (int)m : 32, (int)in_f, (int)out_f);
        Status s = ensure_scratch(pb);
        return s.ok() ? wide_gemm(dtype, w, a, y, m, in_f, out_f, reinterpret_cast<float *>(scratch())) : s;
    }
    Status s = cuda_status(gemv_impl_ == 1   ? launch_gemv_q8(dtype, w, a, y, (int)m, (int)in_f, (int)out_f, nullptr, dev_, stream_)
                           : (dtype == DT_Q4K && gemv_impl_ == 0)
                               ? launch_gemv_q4k_mma(w, &a, nullptr, y, (int)m, (int)in_f, (int)out_f, dev_, status_dev_, stream_)
                               : launch_gemv_stream(dtype, w, a, y, (int)m, (int)in_f, (int)out_f, dev_, status_dev_, stream_),
                           "gemv_q8");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::gemv_q8_pair(int dtype, const uint8_t *w1, float *y1, uint32_t out_f1, const uint8_t *w2, float *y2, uint32_t out_f2,
                                 const Q8Dev &a, uint32_t m, uint32_t in_f) {
    if (dtype == DT_Q4K && gemv_impl_ == 0 && m >= 1 && m <= 8 && in_f && in_f % 256 == 0 && out_f1 && out_f2 && a.gran == 256 &&
        !overlap(y1, (size_t)m * out_f1, y2, (size_t)m * out_f2)) {
        cudaSetDevice(device_);
        Status s = cuda_status(launch_gemv_q4k_mma_pair(w1, y1, (int)out_f1, w2, y2, (int)out_f2, &a, nullptr, (int)m, (int)in_f, dev_, status_dev_, stream_),
                               "gemv_q8_pair");
        if (s.ok()) launches_++;
        return s;
    }
    if (m == 1 && gemv_impl_ == 0 && out_f1 && out_f2 && a.gran == act_gran(dtype) && gemv_row_takes(dtype, (int)in_f) && (dtype != DT_Q6K || in_f <= 36864) &&
        !overlap(y1, out_f1, y2, out_f2)) {
        cudaSetDevice(device_);
        const GemvRowMat mats[2] = {{w1, y1, (int)out_f1, nullptr, (int)out_f2}, {w2, y2, (int)out_f2, nullptr, (int)out_f1}};
        const cudaError_t e = launch_gemv_row(GemvRow{dtype, (int)in_f, mats, 2, &a}, dev_, status_dev_, stream_);
        if (e == cudaSuccess) launches_++;
        if (e != cudaErrorInvalidValue) return cuda_status(e, "gemv_q8_pair");
        cudaGetLastError();
    }
    if (m > 8 && m <= 32 && out_f1 && out_f2 && wide_applies(dtype, m, in_f, (uint64_t)out_f1 + out_f2, INFR_ACT_INT8) && a.gran == 256 && (dtype != DT_Q6K || a.sums16)) {
        if (tc_wins(dtype, m, in_f, (uint64_t)out_f1 + out_f2)) {
            cudaSetDevice(device_);
            return tc_linear(dtype, w1, y1, out_f1, w2, y2, out_f2, nullptr, &a, m, in_f);
        }
        // a few dozen rows: both weights in one launch of the wide GEMV (and one launch that adds the K chunks of both)
        cudaSetDevice(device_);
        Status s = ensure_scratch(gemv_wide_partial_bytes((int)m, (int)in_f, (int)(out_f1 + out_f2)));
        return s.ok() ? wide_gemm(dtype, w1, a, y1, m, in_f, out_f1, reinterpret_cast<float *>(scratch()), w2, y2, out_f2) : s;
    }
    Status s = gemv_q8(dtype, w1, a, y1, m, in_f, out_f1);
    return s.ok() ? gemv_q8(dtype, w2, a, y2, m, in_f, out_f2) : s;
}

// ---- the other ops of a dense decode step ----
Status CudaBackend::rms_norm(const float *a, const float *b, float *sum_dst, const float *w, float *dst, uint32_t rows, uint32_t dim, float eps) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_rms_norm(a, b, sum_dst, w, dst, (int)rows, (int)dim, eps, stream_), "rms_norm");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::rope(const float *x, const int32_t *positions, float *dst, uint32_t rows, uint32_t n_head, uint32_t head_dim,
                         uint32_t rope_dim, float theta, int neox) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_rope(x, positions, dst, (int)rows, (int)n_head, (int)head_dim, (int)rope_dim, theta, neox, dev_, stream_), "rope");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::write_kv(const float *src, void *cache_at_pos, size_t n) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_write_kv_f16(src, cache_at_pos, n, dev_, stream_), "write_kv");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::rope_write_kv(const infr_attn_desc &d, float theta, int neox, float *q, const float *k, const float *v,
                                  const int32_t *positions, void *k_cache, void *v_cache, int write_pos, const int32_t *block_table,
                                  uint32_t table_stride, uint32_t n_pages) {
    cudaSetDevice(device_);
    const uint32_t n_seq = d.n_seq ? d.n_seq : 1;
    Status s = cuda_status(launch_rope_write_kv(q, k, v, positions, k_cache, v_cache, (int)(n_seq * d.rows), (int)d.n_head, (int)d.n_kv,
                                                (int)d.head_dim, theta, neox, (int)d.rows, block_table ? 0 : (size_t)d.seq_stride, dev_, stream_, write_pos, block_table,
                                                (int)table_stride, (int)n_pages),
                           "rope_write_kv");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::rms_norm_q8(const float *a, const float *b, float *sum_dst, const float *w, uint32_t rows, uint32_t dim, float eps, const Q8Dev &q8) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_rms_norm_q8(a, b, sum_dst, w, (int)rows, (int)dim, eps, const_cast<int8_t *>(q8.qs), const_cast<float *>(q8.d),
                                              const_cast<int32_t *>(q8.sums), const_cast<int32_t *>(q8.sums16), stream_),
                           "rms_norm_q8");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::gated_act_q8(const float *gate, const float *up, uint32_t rows, uint32_t nff, const Q8Dev &q8) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_gated_silu_q8(gate, up, (int)rows, (int)nff, const_cast<int8_t *>(q8.qs), const_cast<float *>(q8.d),
                                                const_cast<int32_t *>(q8.sums), const_cast<int32_t *>(q8.sums16), stream_),
                           "gated_act_q8");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::attention(const infr_attn_desc &d, const float *q, const void *k_cache, const void *v_cache, float *dst, const Q8Dev *q8,
                              const int32_t *seq_pos, const int32_t *block_table, uint32_t table_stride, uint32_t n_pages) {
    cudaSetDevice(device_);
    const uint32_t n_seq = d.n_seq ? d.n_seq : 1;
    const size_t ws = attention_workspace_bytes((int)(n_seq * d.rows), (int)d.n_head, (int)d.head_dim, (int)(d.pos + d.rows));
    Status s = ensure_scratch(ws);
    if (!s.ok()) return s;
    s = cuda_status(launch_attention(q, k_cache, v_cache, dst, scratch_, (int)n_seq, (int)d.rows, (int)d.n_head, (int)d.n_kv, (int)d.head_dim,
                                     d.scale, (int)d.pos, block_table ? 0 : (size_t)d.seq_stride, dev_.sm_count, stream_, status_dev_, q8 ? const_cast<int8_t *>(q8->qs) : nullptr,
                                     q8 ? const_cast<float *>(q8->d) : nullptr, q8 ? const_cast<int32_t *>(q8->sums) : nullptr,
                                     q8 ? const_cast<int32_t *>(q8->sums16) : nullptr, seq_pos, block_table, (int)table_stride, (int)n_pages),
                    "attention");
    if (s.ok()) launches_ += 2;
    return s;
}

Status CudaBackend::gated_act(const float *gate, const float *up, float *dst, size_t n) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_gated_silu(gate, up, dst, n, dev_, stream_), "gated_act");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::add(const float *a, const float *b, float *dst, size_t n) {
    cudaSetDevice(device_);
    Status s = cuda_status(launch_add(a, b, dst, n, dev_, stream_), "add");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::argmax(const float *x, uint32_t *dst, uint32_t n, uint32_t rows) {
    cudaSetDevice(device_);
    Status s = ensure_scratch(argmax_workspace_bytes(n, rows));
    if (!s.ok()) return s;
    s = cuda_status(launch_argmax(x, dst, scratch_, n, rows, stream_), "argmax");
    if (s.ok()) launches_ += 2;
    return s;
}

// rows == 1 or `reference`: every expert bank works on raw f32 activations (int8_ok false,
// crates/infr-cpu/src/lib.rs:2359): dequantised weight rows, f32 dot, pairs kept in (row, rank) order.
Status CudaBackend::moe_ffn_f32(const MoeArgs &a) {
    cudaSetDevice(device_);
    const size_t rows = a.rows, ne = a.ne, nff = a.n_ff, nu = a.n_used, nx = a.n_expert;
    const size_t n_pairs = rows * nu;
    if (n_pairs > 65535) return Status::Err(INFR_E_UNSUPPORTED, "moe_ffn (f32 path): more than 65535 routed pairs");
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes, 256);
        return o;
    };
    const size_t o_logits = take(rows * nx * 4), o_ids = take(n_pairs * 4), o_w = take(n_pairs * 4);
    const size_t o_g = take(n_pairs * nff * 4), o_u = take(n_pairs * nff * 4), o_act = take(n_pairs * nff * 4);
    const size_t o_q = take(n_pairs * nff), o_d = take(n_pairs * (nff / 256) * 4), o_s = take(n_pairs * (nff / 32) * 4);
    const size_t o_y = take(n_pairs * ne * 4);
    Status s = ensure_scratch(off);
    if (!s.ok()) return s;
    uint8_t *b = scratch();
    float *logits = a.logits ? a.logits : reinterpret_cast<float *>(b + o_logits);
    int32_t *ids = a.sel_ids ? a.sel_ids : reinterpret_cast<int32_t *>(b + o_ids);
    float *w = a.sel_w ? a.sel_w : reinterpret_cast<float *>(b + o_w);
    float *g = reinterpret_cast<float *>(b + o_g), *u = reinterpret_cast<float *>(b + o_u), *act = reinterpret_cast<float *>(b + o_act);
    float *y = reinterpret_cast<float *>(b + o_y);
    const size_t gu_stride = nff * (ne / 256) * 144, d_stride = ne * (nff / 256) * 144;
#define INFR_STEP(call, what)          \
    do {                               \
        s = cuda_status((call), what); \
        if (!s.ok()) return s;         \
        launches_++;                   \
    } while (0)
    // one decoded token: router, gate and up, down (router_x and x: the row as the router and as the experts see it)
    if (rows == 1 && moe_row_takes((int)ne, (int)nff, (int)nx, (int)nu, a.x, a.router, a.gate, a.up, a.down)) {
        INFR_STEP(launch_moe_router(a.router, a.router_x, logits, (int)rows, (int)ne, (int)nx, dev_, status_dev_, stream_), "moe router");
        INFR_STEP(launch_moe_gate_up_row(logits, a.x, a.gate, a.up, act, ids, w, (int)ne, (int)nff, (int)nx, (int)nu, a.scale, a.norm_w, dev_, stream_),
                  "moe gate, up");
        INFR_STEP(launch_moe_down_row(a.down, act, ids, w, a.dst, (int)ne, (int)nff, (int)nu, dev_, stream_), "moe down");
        return Status::Ok();
    }
    INFR_STEP(launch_moe_router(a.router, a.router_x, logits, (int)rows, (int)ne, (int)nx, dev_, status_dev_, stream_), "moe router");
    INFR_STEP(launch_moe_route(logits, (int)rows, (int)nx, (int)nu, a.scale, a.norm_w, ids, w, stream_), "moe route");
    INFR_STEP(launch_gemv_q4k_f32_sel(a.gate, ids, gu_stride, a.x, (int)nu, g, (int)n_pairs, (int)ne, (int)nff, dev_, stream_), "moe gate f32");
    INFR_STEP(launch_gemv_q4k_f32_sel(a.up, ids, gu_stride, a.x, (int)nu, u, (int)n_pairs, (int)ne, (int)nff, dev_, stream_), "moe up f32");
    INFR_STEP(launch_moe_swiglu_quant(g, u, (int)n_pairs, (int)nff, reinterpret_cast<int8_t *>(b + o_q), reinterpret_cast<float *>(b + o_d),
                                      reinterpret_cast<int32_t *>(b + o_s), nullptr, act, stream_), "moe swiglu");
    INFR_STEP(launch_gemv_q4k_f32_sel(a.down, ids, d_stride, act, 0, y, (int)n_pairs, (int)nff, (int)ne, dev_, stream_), "moe down f32");
    INFR_STEP(launch_moe_combine(y, nullptr, w, (int)rows, (int)nu, (int)ne, a.dst, stream_), "moe combine");
#undef INFR_STEP
    return Status::Ok();
}

// 8-row items to expect of an expert that each of `rows` rows picks with probability p: the sum over k of P(more than 8 k rows).
static double expected_items(double p, int rows) {
    double pmf = std::pow(1.0 - p, rows);
    if (p >= 1.0 || pmf < 1e-30) return (p * rows + 3.5) / 8;  // an item of every expert is half full on average
    double below = 0, sum = 0;
    for (int c = 0; c <= rows; c++) {  // P(c rows) from P(c - 1 rows)
        below += pmf;
        if (1.0 - below < 1e-9) break;
        if (c % 8 == 0) sum += 1.0 - below;
        pmf *= p / (1.0 - p) * (rows - c) / (c + 1);
    }
    return sum;
}

Status CudaBackend::moe_ffn(const MoeArgs &a) {
    auto bank_ok = [](int dt) { return dt == DT_Q4K || dt == DT_Q6K; };
    if (!bank_ok(a.gate_dt) || !bank_ok(a.up_dt) || !bank_ok(a.down_dt))
        return Status::Err(INFR_E_UNSUPPORTED, "moe_ffn: expert banks must be Q4_K or Q6_K");
    const bool any_q6 = a.gate_dt == DT_Q6K || a.up_dt == DT_Q6K || a.down_dt == DT_Q6K;
    if (a.ne == 0 || a.ne % 256 || a.n_ff == 0 || a.n_ff % 256)
        return Status::Err(INFR_E_UNSUPPORTED, fmt("moe_ffn: ne=%u and n_ff_exp=%u must be multiples of 256", a.ne, a.n_ff));
    if (a.n_expert == 0 || a.n_expert > 1024 || a.n_used == 0 || a.n_used > 32 || a.n_used > a.n_expert)
        return Status::Err(INFR_E_INVALID, fmt("moe_ffn: n_expert=%u (<=1024), n_used=%u (<=32)", a.n_expert, a.n_used));
    if (a.rows == 0) return Status::Ok();
    if (((uintptr_t)a.x | (uintptr_t)a.router_x | (uintptr_t)a.router) % 16)  // (rows go by 16-byte loads and bulk copies)
        return Status::Err(INFR_E_INVALID, "moe_ffn: x, router_x and router must be 16-byte aligned");
    if (((size_t)a.rows * a.n_used + 31) / 32 * a.n_expert * 4 > (size_t)200 * 1024)
        return Status::Err(INFR_E_UNSUPPORTED, fmt("moe_ffn: %u rows x %u experts per row exceed what one call sorts (split the rows)", a.rows, a.n_used));
    if (a.rows < 2 || reference_) {
        if (a.n_local != a.n_expert) return Status::Err(INFR_E_UNSUPPORTED, "moe_ffn: a local expert range needs the int8 path (rows >= 2, no reference mode)");
        if (any_q6) return Status::Err(INFR_E_UNSUPPORTED, "moe_ffn: Q6_K expert banks run on the int8 path only (rows >= 2, no reference mode)");
        return moe_ffn_f32(a);
    }
    cudaSetDevice(device_);
    const size_t rows = a.rows, ne = a.ne, nff = a.n_ff, nu = a.n_used, nx = a.n_expert;
    const size_t n_pairs = rows * nu;
    const size_t max_items = n_pairs / 8 + nx + 1;
    // Experts that see a few dozen rows each run on the tensor-memory GEMM in grouped form (one slab of 32 or 64 of an expert's
    // rows per token tile: the expert's weights are unpacked once per slab); with only a handful of rows per expert the 8-row
    // grouped GEMV does less padded work.  An expert's load is that of the whole layer, also on a rank that holds some experts.
    // Measured, us a layer (items / slabs of 32 / of 64), by pairs per expert:
    //   128 experts, 2048 -> 768   9: 181 / 214 / 245, 13: 211 / 219 / 253, 16: 258 / 224 / 257, 28: 390 / 286 / 281, 40: 503 / 395 / 306
    //   60 experts, 2048 -> 1536   11: 164 / 189 / 202, 13: 186 / 190 / 204, 16: 194 / 190 / 207, 28: 328 / 230 / 223
    //   32 experts, 1024 -> 1024   13: 70 / 73 / 78, 16: 81 / 74 / 78, 28: 102 / 77 / 82, 32: 103 / 92 / 81
    //   16 experts, 2048 -> 1024   9: 62 / 75 / 79, 13: 68 / 76 / 79, 16: 73 / 77 / 80, 24: 86 / 77 / 81, 28: 96 / 90 / 82
    //   8 experts, 4096 -> 2048    9: 75 / 90 / 97, 13: 90 / 93 / 98, 16: 96 / 92 / 98, 24: 136 / 108 / 115, 28: 153 / 125 / 115
    //   64 experts, 1024 -> 256    9: 62 / 62 / 67, 13: 64 / 63 / 69, 16: 80 / 65 / 70, 28: 91 / 74 / 76
    // Items lose their lead earlier, from 11 rows an expert on, where rows are long and the weights many (items / slabs of 32, M = 2^20 weights a bank):
    //   32 experts, 3072 -> 1536 (144 M)  10: 161 / 173, 11: 183 / 172;  4096 -> 1536 (192 M)  10: 194 / 211, 11: 223 / 210;  128 experts (768 M)  10: 563 /
    //   601, 12: 709 / 607;  8 experts, 4096 -> 7168 (224 M)  9: 180 / 192, 11: 209 / 192;  64 experts, 2048 -> 5632 (704 M)  11: 511 / 529, 12: 581 / 525
    // and not with shorter rows or fewer weights:
    //   64 experts, 2048 -> 1792 (224 M)  11: 182 / 225, 14: 205 / 223;  128 experts, 2048 -> 1024 (256 M)  11: 255 / 268, 14: 257 / 272;  16 experts,
    //   4096 -> 2048 (128 M)  11: 121 / 142, 14: 141 / 143, 15: 169 / 142;  3072 -> 2048 (96 M)  14: 120 / 128
    // (a layer with a Q6_K bank takes 8-row items throughout: the GEMM's copies want rows of whole 2048-element chunks)
    const size_t bank_weights = a.n_local * ne * nff;
    const bool large = (ne >= 3072 && bank_weights > ((size_t)128 << 20)) || bank_weights >= ((size_t)512 << 20);
    const bool long_rows = !grouped_q4k_takes((int)(ne > nff ? ne : nff), dev_);  // no room for an item's rows
    const bool grouped_gemm = !any_q6 && (mmq_impl_ == 2 || (mmq_impl_ == 0 && (long_rows || 2 * n_pairs >= (size_t)(large ? 21 : 28) * nx)));
    const int slab = n_pairs >= 28 * nx ? 64 : 32;
    const size_t max_slabs = n_pairs / slab + a.n_local + 1;
    // scratch carve-up (all 256-byte aligned)
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes, 256);
        return o;
    };
    const size_t o_logits = take(rows * nx * 4), o_ids = take(n_pairs * 4), o_w = take(n_pairs * 4);
    const size_t o_prow = take(n_pairs * 4), o_pslot = take(n_pairs * 4);
    const size_t o_ie = take(max_items * 4), o_ip = take(max_items * 4), o_ic = take(max_items * 4), o_ni = take(4);
    auto items_only = [&](size_t bytes) { return grouped_gemm ? 0 : take(bytes); };  // (the GEMM's layouts quantise the rows)
    const size_t o_xq = items_only(rows * ne), o_xd = items_only(rows * (ne / 256) * 4), o_xs = items_only(rows * (ne / 32) * 4);
    const size_t o_xs16 = any_q6 ? take(rows * (ne / 16) * 4) : 0, o_as16 = any_q6 ? take(n_pairs * (nff / 16) * 4) : 0;
    const size_t o_g = take(n_pairs * nff * 4), o_u = take(n_pairs * nff * 4);
    const size_t o_aq = items_only(n_pairs * nff), o_ad = items_only(n_pairs * (nff / 256) * 4), o_as = items_only(n_pairs * (nff / 32) * 4);
    const size_t o_y = take(n_pairs * ne * 4);
    const size_t o_px = grouped_gemm ? take(gemm_tc_grouped_record_bytes(slab, (int)max_slabs, (int)ne)) : 0;
    const size_t o_pa = grouped_gemm ? take(gemm_tc_grouped_record_bytes(slab, (int)max_slabs, (int)nff)) : 0;
    Status s = ensure_scratch(off);
    if (!s.ok()) return s;
    uint8_t *b = scratch();
    float *logits = a.logits ? a.logits : reinterpret_cast<float *>(b + o_logits);
    int32_t *ids = a.sel_ids ? a.sel_ids : reinterpret_cast<int32_t *>(b + o_ids);
    float *w = a.sel_w ? a.sel_w : reinterpret_cast<float *>(b + o_w);
    int32_t *prow = reinterpret_cast<int32_t *>(b + o_prow), *pslot = reinterpret_cast<int32_t *>(b + o_pslot);
    int32_t *ie = reinterpret_cast<int32_t *>(b + o_ie), *ip = reinterpret_cast<int32_t *>(b + o_ip);
    int32_t *ic = reinterpret_cast<int32_t *>(b + o_ic), *ni = reinterpret_cast<int32_t *>(b + o_ni);
    int8_t *xq = reinterpret_cast<int8_t *>(b + o_xq);
    float *xd = reinterpret_cast<float *>(b + o_xd);
    int32_t *xs = reinterpret_cast<int32_t *>(b + o_xs);
    float *g = reinterpret_cast<float *>(b + o_g), *u = reinterpret_cast<float *>(b + o_u);
    int8_t *aq = reinterpret_cast<int8_t *>(b + o_aq);
    float *ad = reinterpret_cast<float *>(b + o_ad);
    int32_t *as = reinterpret_cast<int32_t *>(b + o_as);
    float *y = reinterpret_cast<float *>(b + o_y);
#define INFR_STEP(call, what)                       \
    do {                                            \
        s = cuda_status((call), what);              \
        if (!s.ok()) return s;                      \
        launches_++;                                \
    } while (0)
    INFR_STEP(launch_moe_router(a.router, a.router_x, logits, (int)rows, (int)ne, (int)nx, dev_, status_dev_, stream_), "moe router");
    INFR_STEP(launch_moe_route(logits, (int)rows, (int)nx, (int)nu, a.scale, a.norm_w, ids, w, stream_), "moe route");
    INFR_STEP(launch_moe_bucket(ids, (int)rows, (int)nu, (int)nx, (int)a.expert_lo, (int)a.n_local, grouped_gemm ? slab : 8, prow, pslot, ie, ip, ic, ni,
                                nullptr, stream_),
              "moe bucket");
    // stage A: every distinct row quantised once (lib.rs:2688-2718), or by each of its slots where they are laid out for the GEMM (the layout waits on
    // its stores, not on the quantiser, and a launch of 3 us is saved)
    int32_t *xs16 = any_q6 ? reinterpret_cast<int32_t *>(b + o_xs16) : nullptr, *as16 = any_q6 ? reinterpret_cast<int32_t *>(b + o_as16) : nullptr;
    if (!grouped_gemm) INFR_STEP(launch_quantize_q8(a.x, (int)rows, (int)ne, 256, xq, xd, xs, xs16, nullptr, nullptr, stream_), "moe quantize x");
    Q8Dev xa{xq, xd, xs, xs16, 256};
    // one expert bank against the routed rows, 8-row items on the warp matrix unit (Q6_K rows too long for its tiles: byte-dot kernel)
    const int items = (int)((double)a.n_local * expected_items((double)nu / (double)nx, (int)rows) + 0.5);
    auto bank_gemm = [&](int dt, const uint8_t *bank, const Q8Dev &acts, float *out, uint32_t k, uint32_t o, const int32_t *rows_of, const uint8_t *bank2 = nullptr,
                         float *out2 = nullptr) {
        if (dt == DT_Q4K)
            return launch_grouped_q4k_mma(bank, bank2, (int)a.n_local, acts, out, out2, (int)k, (int)o, ie, ip, ic, ni, rows_of, (int)max_items, items, dev_, status_dev_,
                                          stream_);
        const cudaError_t e = launch_grouped_q6_mma(bank, acts, out, (int)k, (int)o, ie, ip, ic, ni, rows_of, (int)max_items, items, dev_, status_dev_, stream_);
        if (e != cudaErrorInvalidValue) return e;
        cudaGetLastError();
        return launch_grouped_q6k(bank, acts, out, (int)k, (int)o, ie, ip, ic, ni, rows_of, (int)max_items, dev_, stream_);
    };
    if (grouped_gemm) {
        // stage B: both banks read the same gathered activation planes (laid out once); stage C; stage D on the
        // re-quantised pairs; stage E
        auto gemm = [&](const uint8_t *bank, const uint8_t *bank2, const uint8_t *rec, float *out, float *out2, uint32_t k, uint32_t o) {
            return launch_gemm_tc_grouped(slab, bank, bank2, (int)a.n_local, rec, out, out2, (int)k, (int)o, ie, ip, ic, ni, (int)max_slabs, dev_, status_dev_, stream_);
        };
        INFR_STEP(launch_gemm_tc_grouped_prep(slab, a.x, b + o_px, (int)ne, ie, ip, ic, ni, prow, (int)max_slabs, stream_), "moe layout x");
        INFR_STEP(gemm(a.gate, a.up, b + o_px, g, u, (uint32_t)ne, (uint32_t)nff), "moe gate, up (grouped gemm)");
        INFR_STEP(launch_gemm_tc_grouped_silu_prep(slab, g, u, b + o_pa, (int)nff, ie, ip, ic, ni, (int)max_slabs, stream_), "moe swiglu, layout");
        INFR_STEP(gemm(a.down, nullptr, b + o_pa, y, nullptr, (uint32_t)nff, (uint32_t)ne), "moe down (grouped gemm)");
        INFR_STEP(launch_moe_combine(y, pslot, w, (int)rows, (int)nu, (int)ne, a.dst, stream_), "moe combine");
        return Status::Ok();
    }
    // stage B: gate and up expert GEMMs, rows gathered per pair
    if (a.gate_dt == DT_Q4K && a.up_dt == DT_Q4K) {
        INFR_STEP(bank_gemm(DT_Q4K, a.gate, xa, g, (uint32_t)ne, (uint32_t)nff, prow, a.up, u), "moe gate, up");
    } else {
        INFR_STEP(bank_gemm(a.gate_dt, a.gate, xa, g, (uint32_t)ne, (uint32_t)nff, prow), "moe gate");
        INFR_STEP(bank_gemm(a.up_dt, a.up, xa, u, (uint32_t)ne, (uint32_t)nff, prow), "moe up");
    }
    // stage C: SwiGLU and re-quantisation per pair
    INFR_STEP(launch_moe_swiglu_quant(g, u, (int)n_pairs, (int)nff, aq, ad, as, as16, nullptr, stream_), "moe swiglu");
    Q8Dev aa{aq, ad, as, as16, 256};
    // stage D: down GEMMs; stage E: rank-order combine
    INFR_STEP(bank_gemm(a.down_dt, a.down, aa, y, (uint32_t)nff, (uint32_t)ne, nullptr), "moe down");
    INFR_STEP(launch_moe_combine(y, pslot, w, (int)rows, (int)nu, (int)ne, a.dst, stream_), "moe combine");
#undef INFR_STEP
    return Status::Ok();
}

Status CudaBackend::gemv_block_acc(int dtype, const uint8_t *w, const float *x, int32_t *acc, uint32_t in_f, uint32_t out_f) {
    if (dtype != DT_Q4K && dtype != DT_Q6K && dtype != DT_Q2_0)
        return Status::Err(INFR_E_UNSUPPORTED, fmt("gemv_block_acc: dtype code %d", dtype));
    const int be = block_elems(dtype);
    if (in_f == 0 || in_f % (uint32_t)be || in_f % 16) return Status::Err(INFR_E_INVALID, fmt("gemv_block_acc: in_f=%u", in_f));
    cudaSetDevice(device_);
    Q8Dev a;
    Status s = quantize_for(dtype, x, 1, in_f, &a);
    if (!s.ok()) return s;
    s = cuda_status(launch_gemv_q8(dtype, w, a, nullptr, 1, (int)in_f, (int)out_f, acc, dev_, stream_), "gemv_block_acc");
    if (s.ok()) launches_++;
    return s;
}

// ------------------------------------------------------------------------------ capture and timing
Status CudaBackend::capture_begin() {
    if (capturing_) return Status::Err(INFR_E_INVALID, "capture_begin: already capturing");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture");
    if (s.ok()) capturing_ = true;
    return s;
}

Status CudaBackend::capture_end(infr_cuda_graph **out) {
    if (!capturing_) return Status::Err(INFR_E_INVALID, "capture_end: not capturing");
    capturing_ = false;
    cudaSetDevice(device_);
    auto *g = new infr_cuda_graph();
    Status s = cuda_status(cudaStreamEndCapture(stream_, &g->graph), "cudaStreamEndCapture");
    if (s.ok()) s = cuda_status(cudaGraphInstantiate(&g->exec, g->graph, 0), "cudaGraphInstantiate");
    if (s.ok()) {
        size_t nn = 0;
        cudaGraphGetNodes(g->graph, nullptr, &nn);
        std::vector<cudaGraphNode_t> nodes(nn);
        if (nn) cudaGraphGetNodes(g->graph, nodes.data(), &nn);
        for (auto nd : nodes) {
            cudaGraphNodeType ty;
            if (cudaGraphNodeGetType(nd, &ty) == cudaSuccess && ty == cudaGraphNodeTypeKernel) g->kernel_nodes++;
        }
    }
    if (!s.ok()) {
        graph_free(g);
        return s;
    }
    *out = g;
    return Status::Ok();
}

Status CudaBackend::graph_launch(infr_cuda_graph *g) {
    if (!g || !g->exec) return Status::Err(INFR_E_INVALID, "graph_launch: null graph");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaGraphLaunch(g->exec, stream_), "cudaGraphLaunch");
    if (s.ok()) launches_ += g->kernel_nodes;
    return s;
}

void CudaBackend::graph_free(infr_cuda_graph *g) {
    if (!g) return;
    cudaSetDevice(device_);
    cudaStreamSynchronize(stream_);
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    delete g;
}

Status CudaBackend::timer_start() {
    cudaSetDevice(device_);
    return cuda_status(cudaEventRecord(ev0_, stream_), "cudaEventRecord");
}

Status CudaBackend::timer_stop(float *ms) {
    if (!ms) return Status::Err(INFR_E_INVALID, "timer_stop: null output");
    cudaSetDevice(device_);
    Status s = cuda_status(cudaEventRecord(ev1_, stream_), "cudaEventRecord");
    if (s.ok()) s = cuda_status(cudaEventSynchronize(ev1_), "cudaEventSynchronize");
    if (s.ok()) s = cuda_status(cudaEventElapsedTime(ms, ev0_, ev1_), "cudaEventElapsedTime");
    return s.ok() ? check_device_status() : s;
}

Status CudaBackend::flush_l2() {
    cudaSetDevice(device_);
    if (!flush_) {
        if (capturing_) return Status::Err(INFR_E_INVALID, "flush_l2: first use during stream capture");
        flush_bytes_ = align_up(dev_.l2_bytes * 2 + (64u << 20), 1 << 20);
        Status s = cuda_status(cudaMalloc(&flush_, flush_bytes_), "flush cudaMalloc");
        if (!s.ok()) return s;
    }
    Status s = cuda_status(launch_fill_u32(static_cast<uint32_t *>(flush_), flush_bytes_ / 4, (uint32_t)launches_, stream_), "flush_l2");
    if (s.ok()) launches_++;
    return s;
}

Status CudaBackend::tensor_peak_i8(uint32_t n_batches, uint32_t launches, float *ms, double *ops) {
    if (!ms || !ops || launches == 0 || launches > 100000 || n_batches == 0 || n_batches > 4096)
        return Status::Err(INFR_E_INVALID, "tensor_peak_i8: 1..4096 batches, 1..100000 launches, non-null outputs");
    if (capturing_) return Status::Err(INFR_E_INVALID, "tensor_peak_i8 during stream capture");
    cudaSetDevice(device_);
    Status s = ensure_scratch(256);
    if (!s.ok()) return s;
    int32_t *check = reinterpret_cast<int32_t *>(scratch());
    if (!(s = cuda_status(cudaMemsetAsync(check, 0xff, 8, stream_), "tensor_peak memset")).ok()) return s;
    // one untimed launch: module load, first tensor-memory allocation
    if (!(s = cuda_status(launch_tensor_peak_i8(n_batches, check, dev_, status_dev_, stream_), "tensor_peak_i8")).ok()) return s;
    if (!(s = cuda_status(cudaEventRecord(ev0_, stream_), "cudaEventRecord")).ok()) return s;
    for (uint32_t i = 0; i < launches; i++)
        if (!(s = cuda_status(launch_tensor_peak_i8(n_batches, check, dev_, status_dev_, stream_), "tensor_peak_i8")).ok()) return s;
    launches_ += launches + 1;
    if (!(s = cuda_status(cudaEventRecord(ev1_, stream_), "cudaEventRecord")).ok()) return s;
    if (!(s = cuda_status(cudaEventSynchronize(ev1_), "cudaEventSynchronize")).ok()) return s;
    if (!(s = cuda_status(cudaEventElapsedTime(ms, ev0_, ev1_), "cudaEventElapsedTime")).ok()) return s;
    if (!(s = check_device_status()).ok()) return s;
    int32_t got[2] = {0, 0};
    if (!(s = cuda_status(cudaMemcpyAsync(got, check, 8, cudaMemcpyDeviceToHost, stream_), "tensor_peak readback")).ok()) return s;
    if (!(s = cuda_status(cudaStreamSynchronize(stream_), "tensor_peak sync")).ok()) return s;
    const int32_t want = tensor_peak_i8_expected(n_batches);
    if (got[0] != want || got[1] != want)
        return Status::Err(INFR_E_CUDA, fmt("tensor_peak_i8: accumulator check failed (got %d and %d, the operand pattern implies %d)", got[0], got[1], want));
    *ops = tensor_peak_i8_ops(n_batches, dev_) * launches;
    return Status::Ok();
}

}  // namespace infr
