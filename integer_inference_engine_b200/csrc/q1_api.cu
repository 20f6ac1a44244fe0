// C-ABI of the Q1_0 dense path (include/iie_q1.h): registry of re-ordered weights, grow-only device
// scratch, host-pointer entries with the reference's names and return codes, and one device-pointer entry.
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <initializer_list>
#include <mutex>
#include <vector>

#include "../../include/iie_q1.h"
#include "../../include/iie_qk.h"
#include "host_threads.h"
#include "kernels.h"

using namespace iie;

namespace {

struct Q1Weight {
    uint8_t *units = nullptr;
    long long out_f = 0, nb = 0;
    unsigned long long max_scale = 0;
    bool sc32 = false;
    bool live = false;
};

std::recursive_mutex q_mu;
std::vector<Q1Weight> q_w;
unsigned long long q_weight_bytes = 0;
cudaStream_t q_stream = nullptr;
int *q_cells = nullptr;                 // device ints: [0] digits of a row, [1] rmsnorm flags, [2..3] largest scale of a matrix being registered, [4] flags of the host call under way, [8..15] digits in use (a DigitRing)
int q_ready = -1;

enum QRole { QR_X, QR_PLANES, QR_WORK, QR_KEYS, QR_VALUES, QR_LOGITS, QR_OUT, QR_GAIN, QR_COUNT };
struct QBuf { void *p = nullptr; size_t cap = 0; };
unsigned long long q_generation = 0;   // changes whenever a scratch buffer is freed: captured graphs hold the old addresses
QBuf q_buf[QR_COUNT];

thread_local int q_err_code = 0;
thread_local char q_err[256] = "ok";

int fail(int code, const char *fmt, ...) {
    q_err_code = code;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(q_err, sizeof(q_err), fmt, ap);
    va_end(ap);
    cudaGetLastError();
    return code;
}
void clear_error() { q_err_code = 0; memcpy(q_err, "ok", 3); }

bool q_init() {
    if (q_ready >= 0) return q_ready == 0;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0 ||
        cudaStreamCreateWithFlags(&q_stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&q_cells, 64) != cudaSuccess || cudaMemset(q_cells, 0, 64) != cudaSuccess) {
        cudaGetLastError(); q_ready = 1; return false;
    }
    q_ready = 0;
    return true;
}

void *q_ensure(int role, size_t bytes) {
    QBuf &b = q_buf[role];
    if (b.p && b.cap >= bytes) return b.p;
    // (the prefill's buffers are in no captured graph: growing them leaves graphs valid)
    if (b.p) { cudaDeviceSynchronize(); cudaFree(b.p); b.p = nullptr; b.cap = 0; if (role < QR_WORK || role > QR_LOGITS) q_generation++; }
    const size_t cap = std::max<size_t>(bytes, 256);
    if (cudaMalloc(&b.p, cap) != cudaSuccess) { cudaGetLastError(); b.p = nullptr; return nullptr; }
    b.cap = cap;
    return b.p;
}

// The prompt call's buffers stay for the next prompt (allocating and freeing them takes a millisecond) up to this many bytes in all, 1400
// rows of the 8B model; those of a longer prompt go with its call.
constexpr size_t PROMPT_KEEP = 512 << 20;
struct PromptBuffers {
    ~PromptBuffers() {
        size_t total = 0;
        for (int role = QR_WORK; role <= QR_LOGITS; role++) total += q_buf[role].cap;
        for (int role = QR_WORK; total > PROMPT_KEEP && role <= QR_LOGITS; role++)
            if (q_buf[role].p) { cudaFree(q_buf[role].p); q_buf[role].p = nullptr; q_buf[role].cap = 0; }
    }
};

// The cell that receives the digits in use of the next digit planes, and the one that their kernel clears (null: not to be had).
PlaneDuties next_digits(cudaStream_t s) {
    static DigitRing ring;
    PlaneDuties d;
    if (!ring.next(q_cells + 8, s, d.nl, d.nl_clear)) d.nl = nullptr;
    return d;
}

// Products of rows whose digit planes a kernel `write(duties)` is about to leave in `planes`.  Where the products add
// shares of a tile to their outputs, that kernel clears them, unless they lie over something it reads ([in, in + in_n) or
// [in2, in2 + in_n)): then they are cleared behind it.
template <typename Write>
bool planes_and_products(Write write, const Q1Part *parts, int n, bool sc32, long long nb, const int8_t *planes, long long T, long long frac,
                         const int64_t *in, const int64_t *in2, long long in_n, cudaStream_t s) {
    PlaneDuties d = next_digits(s);
    if (!d.nl) return false;
    bool fused = true;
    long long row_tiles = 0;
    for (int i = 0; i < n; i++) row_tiles += (parts[i].out_f + 127) / 128;
    const bool clear = q1_tc_split(row_tiles, T);
    for (int i = 0; clear && i < n; i++) {
        const Q1Part &p = parts[i];
        const int64_t *end = p.out + T * p.out_f;
        fused = fused && p.add != p.out && (i == 0 || p.out == d.zero + d.zero_n) && (end <= in || in + in_n <= p.out) &&
                (!in2 || end <= in2 || in2 + in_n <= p.out);
        if (i == 0) d.zero = p.out;
        d.zero_n += T * p.out_f;
    }
    if (!clear || !fused) { d.zero = nullptr; d.zero_n = 0; }
    if (write(d) != cudaSuccess) return false;
    for (int i = 0; clear && !fused && i < n; i++)
        if (parts[i].add != parts[i].out && cudaMemsetAsync(parts[i].out, 0, (size_t)T * parts[i].out_f * 8, s) != cudaSuccess) return false;
    return launch_q1_apply(parts, n, sc32, nb, planes, T, frac, d.nl, s) == cudaSuccess;
}

// Products of a single row.  A row that the kernel cannot read in place (misaligned, or under one of the outputs) is copied first.
bool row_products(const Q1Part *parts, int n, bool sc32, long long nb, Q1RowInput in, bool swiglu, long long frac, cudaStream_t s) {
    const long long K = nb * 128;
    bool copy = (reinterpret_cast<uintptr_t>(in.x) & 15) != 0;
    for (int i = 0; i < n; i++) copy = copy || (parts[i].out < in.x + K && in.x < parts[i].out + parts[i].out_f);
    if (copy) {
        int64_t *own = (int64_t *)q_ensure(QR_PLANES, (size_t)K * 8);
        if (!own || cudaMemcpyAsync(own, in.x, (size_t)K * 8, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return false;
        in.x = own;
    }
    return launch_q1_row(parts, n, sc32, nb, in, swiglu, frac, s) == cudaSuccess;
}

bool valid(long long h) { return h >= 0 && (size_t)h < q_w.size() && q_w[(size_t)h].live; }

// upload + re-order; scale_bits is the width of the caller's scale array
long long register_any(const unsigned char *bits, const void *scale, int scale_bits, long long out_f, long long nb, bool keep) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!bits || !scale || out_f <= 0 || nb <= 0) { fail(1, "q1 register: bad arguments"); return -1; }
    if (!q_init()) { fail(2, "q1 register: no usable CUDA device"); return -1; }
    const size_t bsz = (size_t)out_f * nb * 16, ssz = (size_t)out_f * nb * (scale_bits / 8);
    bool sc32 = scale_bits == 32;
    if (!sc32) {
        sc32 = true;
        const long long *s64 = (const long long *)scale;
        for (size_t i = 0; i < (size_t)out_f * nb; i++)
            if (s64[i] > 0x7FFFFFFFLL || s64[i] < -0x80000000LL) { sc32 = false; break; }
    }
    const long long n_tiles = (out_f + 15) / 16;
    const size_t usz = (size_t)n_tiles * nb * q1_unit_bytes(sc32);
    uint8_t *dbits = nullptr, *dscale = nullptr, *units = nullptr;
    bool ok = cudaMalloc(&dbits, bsz) == cudaSuccess && cudaMalloc(&dscale, ssz) == cudaSuccess &&
              cudaMalloc(&units, usz) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(dbits, bits, bsz, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(dscale, scale, ssz, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    unsigned long long *max_cell = (unsigned long long *)(q_cells + 2), max_scale = 0;
    ok = ok && cudaMemsetAsync(max_cell, 0, 8, q_stream) == cudaSuccess &&
         launch_q1_repack(dbits, dscale, scale_bits, sc32, out_f, nb, units, max_cell, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(&max_scale, max_cell, 8, cudaMemcpyDeviceToHost, q_stream) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(q_stream) == cudaSuccess;
    if (dbits) cudaFree(dbits);
    if (dscale) cudaFree(dscale);
    if (!ok) { if (units) cudaFree(units); fail(2, "q1 register: CUDA failure"); return -1; }
    Q1Weight w;
    w.units = units; w.out_f = out_f; w.nb = nb; w.max_scale = max_scale; w.sc32 = sc32; w.live = true;
    q_w.push_back(w);
    if (keep) q_weight_bytes += bsz + ssz;
    return (long long)q_w.size() - 1;
}

// product of device-resident x with weight w into device out; returns 0 / 2 / 4
int apply_device(const Q1Weight &w, const int64_t *xd, long long T, long long frac, int64_t *outd, int max_digits,
                 cudaStream_t s) {
    const long long K = w.nb * 128;
    int8_t *planes = T > 1 || max_digits < 8 ? (int8_t *)q_ensure(QR_PLANES, (size_t)T * 8 * K) : nullptr;
    if (!planes && (T > 1 || max_digits < 8)) return 2;
    const Q1Part part = {w.units, w.out_f, outd, nullptr, w.max_scale};
    int used = 0;
    auto write = [&](const PlaneDuties &d) {
        PlaneDuties dd = d;
        if (max_digits < 8 && !dd.nl) dd.nl = q_cells;
        cudaError_t e = max_digits < 8 ? cudaMemsetAsync(dd.nl, 0, sizeof(int), s) : cudaSuccess;
        if (e == cudaSuccess) e = launch_q1_prep(xd, T, w.nb, planes, dd, s);
        if (e == cudaSuccess && max_digits < 8) e = cudaMemcpyAsync(&used, dd.nl, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && max_digits < 8) e = cudaStreamSynchronize(s);
        return e == cudaSuccess && used > max_digits ? cudaErrorInvalidValue : e;
    };
    bool ok;
    if (T > 1) ok = planes_and_products(write, &part, 1, w.sc32, w.nb, planes, T, frac, xd, nullptr, T * K, s);
    else ok = (max_digits >= 8 || write(PlaneDuties()) == cudaSuccess) && row_products(&part, 1, w.sc32, w.nb, {xd, false, nullptr, 0}, false, frac, s);
    if (ok) return 0;
    return used > max_digits ? 4 : 2;
}

// Result and flag word to the host behind one wait, results of up to 256 KB through page-locked memory (a copy to pageable memory and
// one more for the flag word take 3 to 8 us longer).  False on a CUDA failure and where a kernel's wait gave up.
constexpr size_t STAGE = 256 << 10;
uint8_t *q_stage = nullptr;
bool q_stage_tried = false;
uint8_t *staging() {
    if (!q_stage_tried) {
        q_stage_tried = true;
        if (cudaHostAlloc(&q_stage, STAGE + 64, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); q_stage = nullptr; }
    }
    return q_stage;
}
bool download_checked(void *dst, const void *src, size_t n) {
    staging();
    const bool staged = q_stage && n <= STAGE;
    int pageable = 0;
    int *seen = q_stage ? reinterpret_cast<int *>(q_stage) : &pageable;
    const int *flags = shared_flag_word();
    if (!flags || cudaMemcpyAsync(seen, flags, sizeof(int), cudaMemcpyDeviceToHost, q_stream) != cudaSuccess ||
        cudaMemcpyAsync(staged ? q_stage + 64 : dst, src, n, cudaMemcpyDeviceToHost, q_stream) != cudaSuccess ||
        cudaStreamSynchronize(q_stream) != cudaSuccess) return false;
    if (*seen & FLAG_GAVE_UP) {                        // goes with the call that reports it; the other bits are device-pointer callers'
        const int f = iie_flags_read_clear(q_stream);
        restore_flag_bits(f & ~FLAG_GAVE_UP);
        return false;
    }
    if (staged) memcpy(dst, q_stage + 64, n);
    return true;
}

int apply_host(const Q1Weight &w, const long long *x, long long T, long long frac, long long *out, int max_digits) {
    const size_t xsz = (size_t)T * w.nb * 128 * 8, osz = (size_t)T * w.out_f * 8;
    int64_t *xd = (int64_t *)q_ensure(QR_X, xsz), *od = (int64_t *)q_ensure(QR_OUT, osz);
    if (!xd || !od) return 2;
    if (cudaMemcpyAsync(xd, x, xsz, cudaMemcpyHostToDevice, q_stream) != cudaSuccess) return 2;
    const int rc = apply_device(w, xd, T, frac, od, max_digits, q_stream);
    if (rc != 0) { cudaStreamSynchronize(q_stream); return rc; }
    return download_checked(out, od, osz) ? 0 : 2;
}

int one_shot(const long long *x, const unsigned char *bits, const long long *scale, long long tokens, long long out_f,
             long long nb, long long frac, long long *out, int max_digits) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!x || !bits || !scale || !out || tokens <= 0 || out_f <= 0 || nb <= 0) return fail(1, "q1 linear: bad arguments");
    const long long h = register_any(bits, scale, 64, out_f, nb, false);
    if (h < 0) return q_err_code == 1 ? 1 : 2;
    int rc = apply_host(q_w[(size_t)h], (const long long *)x, tokens, frac, out, max_digits);
    cudaFree(q_w[(size_t)h].units);
    q_w.pop_back();                                    // the temporary registration was the last entry
    if (rc == 2) return fail(2, "q1 linear: CUDA failure");
    if (rc == 4) return fail(4, "q1 linear: an activation needs more digits than the caller allowed");
    return 0;
}

}  // namespace

extern "C" int bonsai_gpu_abi_version(void) { return 3; }
extern "C" int bonsai_gpu_last_error_code(void) { return q_err_code; }
extern "C" const char *bonsai_gpu_last_error(void) { return q_err; }

extern "C" int bonsai_gpu_available(void) {
    int n = 0;
    const cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) cudaGetLastError();
    return (e == cudaSuccess && n > 0) ? 0 : 1;
}

extern "C" int bonsai_gpu_mem_info(unsigned long long *free_bytes, unsigned long long *total_bytes) {
    if (!free_bytes || !total_bytes) return 1;
    size_t f = 0, t = 0;
    if (cudaFree(0) != cudaSuccess || cudaMemGetInfo(&f, &t) != cudaSuccess) { cudaGetLastError(); return 2; }
    *free_bytes = f; *total_bytes = t;
    return 0;
}

extern "C" unsigned long long bonsai_q1_resident_weight_bytes(void) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    return q_weight_bytes;
}

extern "C" int bonsai_q1_linear_gpu(const long long *x, const unsigned char *bits, const long long *scale, long long tokens,
                                    long long out_f, long long n_blocks, long long frac, long long *out) {
    const int rc = one_shot(x, bits, scale, tokens, out_f, n_blocks, frac, out, 8);
    return rc == 0 ? 0 : 1;                            // the reference reports every failure of this entry as 1
}

extern "C" int bonsai_q1_linear_dp4a_gpu(const long long *x, const unsigned char *bits, const long long *scale,
                                         long long tokens, long long out_f, long long n_blocks, long long frac, int L,
                                         long long *out) {
    const int LL = L < 0 ? -L : L;
    if (LL < 1 || LL > 8) return 1;
    return one_shot(x, bits, scale, tokens, out_f, n_blocks, frac, out, LL);
}

extern "C" long long bonsai_q1_register_weight(const unsigned char *bits, const long long *scale, long long out_f,
                                               long long n_blocks) {
    return register_any(bits, scale, 64, out_f, n_blocks, true);
}
extern "C" long long bonsai_q1_register_weight_i32(const unsigned char *bits, const int *scale, long long out_f,
                                                   long long n_blocks) {
    return register_any(bits, scale, 32, out_f, n_blocks, true);
}
extern "C" long long bonsai_q1_register_weight_i32_gpu_layout(const unsigned char *bits, const int *scale, long long out_f,
                                                              long long n_blocks) {
    return register_any(bits, scale, 32, out_f, n_blocks, true);
}
extern "C" long long bonsai_q1_register_weight_i32_bmma(const unsigned char *bits, const int *scale, long long out_f,
                                                        long long n_blocks) {
    return register_any(bits, scale, 32, out_f, n_blocks, true);
}

extern "C" int bonsai_q1_apply_resident(long long handle, const long long *x, long long tokens, long long frac,
                                        long long *out) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!valid(handle) || !x || !out || tokens <= 0) return fail(1, "q1 apply: bad arguments");
    const int rc = apply_host(q_w[(size_t)handle], x, tokens, frac, out, 8);
    if (rc != 0) { fail(rc, "q1 apply: CUDA failure"); return 1; }
    return 0;
}

static void q1_release_model_state();
static void free_host_pool();

extern "C" void bonsai_q1_free_weights(void) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (q_ready == 0) cudaDeviceSynchronize();
    for (auto &w : q_w) if (w.live && w.units) cudaFree(w.units);
    q_w.clear();
    q_weight_bytes = 0;
    for (auto &b : q_buf) if (b.p) { cudaFree(b.p); b.p = nullptr; b.cap = 0; q_generation++; }
    free_host_pool();
    q1_release_model_state();                      // uploaded gain / table buffers and decode contexts name these weights
}

extern "C" int bonsai_rmsnorm_gpu(const long long *x, long long rows, long long cols, long long frac, long long eps,
                                  const long long *gain, long long *out) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!x || !out || rows < 0 || cols <= 0 || frac < 0 || frac > 62 || eps < 0) return fail(1, "rmsnorm: bad arguments");
    if (rows == 0) return 0;
    if (!q_init()) return fail(1, "rmsnorm: no usable CUDA device");
    const size_t xsz = (size_t)rows * cols * 8;
    int64_t *xd = (int64_t *)q_ensure(QR_X, xsz), *od = (int64_t *)q_ensure(QR_OUT, xsz), *gd = nullptr;
    if (!xd || !od) return fail(1, "rmsnorm: out of device memory");
    if (gain && !(gd = (int64_t *)q_ensure(QR_GAIN, (size_t)cols * 8))) return fail(1, "rmsnorm: out of device memory");
    int *flags = q_cells + 1;
    int f = 0;
    bool ok = cudaMemcpyAsync(xd, x, xsz, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    ok = ok && (!gain || cudaMemcpyAsync(gd, gain, (size_t)cols * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess);
    ok = ok && cudaMemsetAsync(flags, 0, sizeof(int), q_stream) == cudaSuccess;
    ok = ok && launch_rmsnorm(xd, rows, cols, gd, (int)frac, (unsigned long long)eps, od, flags, q_stream) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(&f, flags, sizeof(int), cudaMemcpyDeviceToHost, q_stream) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(q_stream) == cudaSuccess;
    if (!ok) return fail(1, "rmsnorm: CUDA failure");
    if (f) return fail(4, "rmsnorm: a row left the exact envelope");
    if (cudaMemcpy(out, od, xsz, cudaMemcpyDeviceToHost) != cudaSuccess) return fail(1, "rmsnorm: CUDA failure");
    return 0;
}

extern "C" int iie_q1_apply_dev(long long handle, const int64_t *x_dev, long long tokens, long long frac, int64_t *out_dev,
                                void *stream) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid(handle) || !x_dev || !out_dev || tokens <= 0) return 1;
    return apply_device(q_w[(size_t)handle], x_dev, tokens, frac, out_dev, 8, (cudaStream_t)stream);
}

extern "C" int iie_q1_apply_fused_dev(long long handle, int mode, const int64_t *x_dev, const int64_t *x2_dev, long long ld,
                                      const int64_t *gain_dev, long long tokens, long long frac, const int64_t *add_dev,
                                      int64_t *out_dev, void *stream) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid(handle) || !x_dev || !out_dev || tokens <= 0 || mode < 0 || mode > 2 || frac < 1 || frac > 29) return 1;
    const Q1Weight &w = q_w[(size_t)handle];
    const long long K = w.nb * 128, T = tokens;
    cudaStream_t s = (cudaStream_t)stream;
    if (mode == 2 && (!x2_dev || ld < K)) return 1;
    int8_t *planes = (int8_t *)q_ensure(QR_PLANES, (size_t)T * 8 * K);
    if (!planes) return 2;
    int *flags = iie::shared_flag_word();
    if (!flags) return 2;
    const Q1Part part = {w.units, w.out_f, out_dev, add_dev, w.max_scale};
    if (T == 1) {
        const int64_t *x = x_dev;
        if (mode == 2) {
            x = (const int64_t *)planes;                               // 8 K bytes: the row itself in place of its digit planes
            if (launch_q1_silu_mul(x_dev, x2_dev, K, (int)frac, (int64_t *)planes, s) != cudaSuccess) return 2;
        }
        return row_products(&part, 1, w.sc32, w.nb, {x, mode == 1, mode == 1 ? gain_dev : nullptr, 1ULL}, false, frac, s) ? 0 : 2;
    }
    auto write = [&](const PlaneDuties &d) {
        if (mode == 1) return iie::launch_rmsnorm_planes(x_dev, T, K, gain_dev, (int)frac, 1ULL, nullptr, planes, flags, d, s);
        if (mode == 2) return iie::launch_q1_prep_swiglu(x_dev, x2_dev, ld, (int)frac, T, w.nb, planes, d, s);
        return iie::launch_q1_prep(x_dev, T, w.nb, planes, d, s);
    };
    return planes_and_products(write, &part, 1, w.sc32, w.nb, planes, T, frac, x_dev, mode == 2 ? x2_dev : gain_dev,
                               mode == 2 ? (T - 1) * ld + K : T * K, s) ? 0 : 2;
}

// One layer of a decode token: norm + Q/K/V product; attention with the per-head norms; O product with the residual; norm + gate/up
// products + SwiGLU; down product with the residual.  Five launches, each started while the one before it runs and waiting for it
// behind the requests for its weights.
static int decode_layer(bool behind, long long wqkv, long long wo, long long w1u, long long w2, const int64_t *n1, const int64_t *n2,
                                       const int64_t *qn, const int64_t *kn, int64_t *x, int64_t *qkv, int64_t *qkvn, int64_t *att, int64_t *h,
                                       int32_t *kcache, int32_t *vcache, long long pos, const int *pos_dev, const int64_t *cos, const int64_t *sin,
                                       int n_heads, int n_kv, int head_dim, long long cache_rows, long long frac, long long inv_sqrt, void *stream) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid(wqkv) || !valid(wo) || !valid(w1u) || !valid(w2) || !n1 || !n2 || !qn || !kn || !x || !qkv || !qkvn || !att || !h || !kcache ||
        !vcache || !cos || !sin || n_heads <= 0 || n_kv <= 0 || head_dim <= 0 || n_heads % n_kv || cache_rows <= 0 || pos < 0 || frac < 1 || frac > 29) return 1;
    const Q1Weight &a = q_w[(size_t)wqkv], &o = q_w[(size_t)wo], &g = q_w[(size_t)w1u], &dn = q_w[(size_t)w2];
    const long long qd = (long long)n_heads * head_dim, kd = (long long)n_kv * head_dim, ffn = dn.nb * 128;
    if (a.out_f != qd + 2 * kd || o.nb * 128 != qd || o.out_f != a.nb * 128 || g.nb != a.nb || g.out_f != 2 * ffn || dn.out_f != o.out_f) return 1;
    cudaStream_t s = (cudaStream_t)stream;
    const int f = (int)frac;
    int *flags = iie::shared_flag_word();
    if (!flags) return 2;
    const Q1Part pa = {a.units, a.out_f, qkv, nullptr, a.max_scale}, po = {o.units, o.out_f, x, x, o.max_scale}, pd = {dn.units, dn.out_f, x, x, dn.max_scale};
    if (!row_products(&pa, 1, a.sc32, a.nb, {x, true, n1, 1ULL, behind}, false, frac, s)) return 2;
    int rc = attn_decode_normed(qkv, qkv + qd, qkv + qd + kd, kcache, vcache, pos, pos_dev, cos, sin, 2, n_heads, n_kv, head_dim, cache_rows, f,
                                inv_sqrt, qn, kn, 1ULL, att, s);
    if (rc == 3)                                       // contexts and head shapes beyond the one-launch form
        rc = launch_rmsnorm_pair(qkv, n_heads, n_kv, head_dim, qn, kn, f, 1ULL, qkvn, flags, s) == cudaSuccess
                 ? iie_attn_decode_dev(qkvn, qkvn + qd, qkv + qd + kd, kcache, vcache, pos, pos_dev, 0, cos, sin, 2, n_heads, n_kv, head_dim,
                                       cache_rows, f, inv_sqrt, att, stream) : 2;
    if (rc != 0) return rc;
    if (!row_products(&po, 1, o.sc32, o.nb, {att, false, nullptr, 0}, false, frac, s)) return 2;
    const size_t up_at = (size_t)(ffn / 16) * g.nb * q1_unit_bytes(g.sc32);          // the rows of the up matrix follow the gate's
    const Q1Part gu[2] = {{g.units, ffn, h, nullptr, g.max_scale}, {g.units + up_at, ffn, h, nullptr, g.max_scale}};
    if (g.nb <= 32) {
        if (!row_products(gu, 2, g.sc32, g.nb, {x, true, n2, 1ULL, true}, true, frac, s)) return 2;
    } else {
        const Q1Part both = {g.units, g.out_f, h, nullptr, g.max_scale};
        if (!row_products(&both, 1, g.sc32, g.nb, {x, true, n2, 1ULL, true}, false, frac, s) ||
            launch_q1_silu_mul(h, h + ffn, ffn, f, h, s) != cudaSuccess) return 2;
    }
    return row_products(&pd, 1, dn.sc32, dn.nb, {h, false, nullptr, 0}, false, frac, s) ? 0 : 2;
}

extern "C" int iie_q1_decode_layer_dev(long long wqkv, long long wo, long long w1u, long long w2, const int64_t *n1, const int64_t *n2,
                                       const int64_t *qn, const int64_t *kn, int64_t *x, int64_t *qkv, int64_t *qkvn, int64_t *att, int64_t *h,
                                       int32_t *kcache, int32_t *vcache, long long pos, const int *pos_dev, const int64_t *cos, const int64_t *sin,
                                       int n_heads, int n_kv, int head_dim, long long cache_rows, long long frac, long long inv_sqrt, void *stream) {
    return decode_layer(false, wqkv, wo, w1u, w2, n1, n2, qn, kn, x, qkv, qkvn, att, h, kcache, vcache, pos, pos_dev, cos, sin, n_heads, n_kv, head_dim,
                        cache_rows, frac, inv_sqrt, stream);
}
extern "C" int iie_q1_decode_layer_behind_dev(long long wqkv, long long wo, long long w1u, long long w2, const int64_t *n1, const int64_t *n2,
                                              const int64_t *qn, const int64_t *kn, int64_t *x, int64_t *qkv, int64_t *qkvn, int64_t *att, int64_t *h,
                                              int32_t *kcache, int32_t *vcache, long long pos, const int *pos_dev, const int64_t *cos, const int64_t *sin,
                                              int n_heads, int n_kv, int head_dim, long long cache_rows, long long frac, long long inv_sqrt, void *stream) {
    return decode_layer(true, wqkv, wo, w1u, w2, n1, n2, qn, kn, x, qkv, qkvn, att, h, kcache, vcache, pos, pos_dev, cos, sin, n_heads, n_kv, head_dim,
                        cache_rows, frac, inv_sqrt, stream);
}

extern "C" int iie_q1_head_norm_dev(const int64_t *x_dev, long long rows_a, long long rows_b, long long width, const int64_t *gain_a_dev,
                                    const int64_t *gain_b_dev, long long frac, int64_t *out_dev, void *stream) {
    if (!x_dev || !out_dev || rows_a < 0 || rows_b < 0 || rows_a + rows_b <= 0 || width <= 0 || frac < 1 || frac > 29) return 1;
    int *flags = iie::shared_flag_word();
    if (!flags) return 2;
    return iie::launch_rmsnorm_pair(x_dev, rows_a, rows_b, width, gain_a_dev, gain_b_dev, (int)frac, 1ULL, out_dev, flags,
                                    (cudaStream_t)stream) == cudaSuccess ? 0 : 2;
}

// Page-locked arrays for results that the caller hands on: a small pool, each array given back when its last user drops it.
namespace {
constexpr size_t HOST_POOL = 64 << 20;         // bytes of the pool at most, in use and free
struct HostArray { void *p; size_t cap; bool used; };
std::mutex h_mu;
std::vector<HostArray> h_pool;
}  // namespace
extern "C" void *iie_host_take(unsigned long long bytes) {
    std::lock_guard<std::mutex> lk(h_mu);
    if (bytes == 0 || bytes > HOST_POOL) return nullptr;
    size_t total = 0;
    for (auto &h : h_pool) {
        if (!h.used && h.cap >= bytes && h.cap <= 2 * bytes) { h.used = true; return h.p; }
        total += h.cap;
    }
    for (size_t i = 0; i < h_pool.size() && total + bytes > HOST_POOL;) {          // free arrays make room
        if (h_pool[i].used) { i++; continue; }
        total -= h_pool[i].cap;
        cudaFreeHost(h_pool[i].p);
        h_pool.erase(h_pool.begin() + (long)i);
    }
    void *p = nullptr;
    try { h_pool.reserve(h_pool.size() + 1); } catch (...) { return nullptr; }
    if (total + bytes > HOST_POOL || cudaHostAlloc(&p, bytes, cudaHostAllocDefault) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    h_pool.push_back({p, (size_t)bytes, true});
    return p;
}
static void free_host_pool() {                           // but for the arrays in use
    std::lock_guard<std::mutex> lk(h_mu);
    for (size_t i = 0; i < h_pool.size();) {
        if (h_pool[i].used) { i++; continue; }
        cudaFreeHost(h_pool[i].p);
        h_pool.erase(h_pool.begin() + (long)i);
    }
}
extern "C" void iie_host_give(void *p) {
    std::lock_guard<std::mutex> lk(h_mu);
    for (auto &h : h_pool) if (h.p == p) h.used = false;
}

extern "C" unsigned long long iie_q1_workspace_generation(void) { return q_generation; }
extern "C" void iie_q1_set_stream(int) {}             // single-row products have one form: the weights always come by bulk copies

extern "C" int iie_q1_silu_mul_dev(const int64_t *gate_dev, const int64_t *up_dev, long long n, long long frac, int64_t *out_dev,
                                   void *stream) {
    if (!gate_dev || !up_dev || !out_dev || n <= 0 || frac < 1 || frac > 29) return 1;
    return iie::launch_q1_silu_mul(gate_dev, up_dev, n, (int)frac, out_dev, (cudaStream_t)stream) == cudaSuccess ? 0 : 2;
}

extern "C" int iie_q1_embed_dev(long long handle, const int *row_dev, long long row, int64_t *out_dev, void *stream) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid(handle) || !out_dev) return 1;
    const Q1Weight &w = q_w[(size_t)handle];
    if (!row_dev && (row < 0 || row >= w.out_f)) return 1;
    return iie::launch_q1_embed_row(w.units, w.sc32, w.nb, row_dev, row, out_dev, (cudaStream_t)stream) == cudaSuccess ? 0 : 2;
}

extern "C" int iie_q1_weight_shape(long long handle, long long *out_f, long long *n_blocks, int *scale_bits) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid(handle)) return 1;
    const Q1Weight &w = q_w[(size_t)handle];
    if (out_f) *out_f = w.out_f;
    if (n_blocks) *n_blocks = w.nb;
    if (scale_bits) *scale_bits = w.sc32 ? 32 : 64;
    return 0;
}

// ====================================================================================================
// Whole-model entries of the 1-bit decoder (bonsai/tools/bonsai_q1_gpu.cu:2020-2030 buffers, 2475-2597 standalone
// attention, 3517-3657 decode context, 3694-3819 prefill forward; bridge bonsai/src/trinote/infer_int/gpu_native.py:
// 418-595).  Same names, argument lists and return codes; the layers run on this library's kernels: RMSNorm fused with
// the digit planes of the following products, Q1_0 products with the residual added in their epilogue, per-head
// norms, rotate-half RoPE + K/V append + exact attention (the attention entries of include/iie_qk.h, rope mode 2),
// wrapping SwiGLU fused with the digit planes of the down product.  K/V rows are kept as int32: a value that does
// not fit, like any RMSNorm envelope miss, gives the overflow status (4, or 2 for the standalone attention entries)
// on which the reference bridge redoes the call on the host.
// ====================================================================================================
namespace {

struct DevBuf { int64_t *p = nullptr; size_t n = 0; };
std::vector<DevBuf> q_bufs;
bool valid_buf(long long h, size_t at_least) { return h >= 0 && (size_t)h < q_bufs.size() && q_bufs[(size_t)h].p && q_bufs[(size_t)h].n >= at_least; }

struct Q1Stack {
    long long n_layers = 0, H = 0, Hkv = 0, hd = 0, d = 0, dff = 0, frac = 0, inv_sqrt = 0;
    unsigned long long eps = 1;
    std::vector<long long> wq, wk, wv, wo, w1, wu, w2, n1g, n2g, qng, kng;
    long long finalg = -1, out_head = -1, cos_h = -1, sin_h = -1;
};

bool shaped(long long h, long long out_f, long long in_f) {
    return valid(h) && q_w[(size_t)h].out_f == out_f && q_w[(size_t)h].nb * 128 == in_f;
}

// every handle of the stack names a live tensor of the right shape; rope tables cover `positions` rows
bool stack_ok(const Q1Stack &m, long long positions) {
    if (m.n_layers <= 0 || m.H <= 0 || m.Hkv <= 0 || m.hd <= 0 || m.d <= 0 || m.dff <= 0 || m.H % m.Hkv || m.hd % 2 || m.d % 128 ||
        m.dff % 128 || (m.H * m.hd) % 128 || m.frac < 1 || m.frac > 29 || !attn_shape_ok((int)m.H, (int)m.Hkv, (int)m.hd)) return false;
    const long long qd = m.H * m.hd, kd = m.Hkv * m.hd;
    for (long long li = 0; li < m.n_layers; li++) {
        const size_t i = (size_t)li;
        if (!shaped(m.wq[i], qd, m.d) || !shaped(m.wk[i], kd, m.d) || !shaped(m.wv[i], kd, m.d) || !shaped(m.wo[i], m.d, qd) ||
            !shaped(m.w1[i], m.dff, m.d) || !shaped(m.wu[i], m.dff, m.d) || !shaped(m.w2[i], m.d, m.dff) ||
            !valid_buf(m.n1g[i], (size_t)m.d) || !valid_buf(m.n2g[i], (size_t)m.d) || !valid_buf(m.qng[i], (size_t)m.hd) ||
            !valid_buf(m.kng[i], (size_t)m.hd)) return false;
    }
    const size_t table = (size_t)positions * (size_t)(m.hd / 2);
    return valid(m.out_head) && q_w[(size_t)m.out_head].nb * 128 == m.d && valid_buf(m.finalg, (size_t)m.d) &&
           valid_buf(m.cos_h, table) && valid_buf(m.sin_h, table);
}

void fill_stack(Q1Stack &m, const long long *wq, const long long *wk, const long long *wv, const long long *wo, const long long *w1,
                const long long *wu, const long long *w2, const long long *n1g, const long long *n2g, const long long *qng,
                const long long *kng) {
    const size_t n = (size_t)m.n_layers;
    m.wq.assign(wq, wq + n); m.wk.assign(wk, wk + n); m.wv.assign(wv, wv + n); m.wo.assign(wo, wo + n); m.w1.assign(w1, w1 + n);
    m.wu.assign(wu, wu + n); m.w2.assign(w2, w2 + n); m.n1g.assign(n1g, n1g + n); m.n2g.assign(n2g, n2g + n);
    m.qng.assign(qng, qng + n); m.kng.assign(kng, kng + n);
}

// activation rows of `rows` tokens, one allocation
struct Work {
    void *base = nullptr;
    int64_t *x = nullptr, *q = nullptr, *k = nullptr, *v = nullptr, *qn = nullptr, *kn = nullptr, *att = nullptr, *g = nullptr, *u = nullptr;
};
bool alloc_work(Work &w, const Q1Stack &m, long long rows, bool keep) {
    const size_t qd = (size_t)(m.H * m.hd), kd = (size_t)(m.Hkv * m.hd), T = (size_t)rows;
    const size_t n = T * ((size_t)m.d + 3 * qd + 3 * kd + 2 * (size_t)m.dff);
    int64_t *p = keep ? (int64_t *)q_ensure(QR_WORK, n * 8) : nullptr;      // kept between calls, or the caller's
    if (!keep) {
        if (cudaMalloc(&w.base, n * 8) != cudaSuccess) { cudaGetLastError(); w.base = nullptr; return false; }
        p = (int64_t *)w.base;
    }
    if (!p) return false;
    // q, k, v and g, u side by side: one range each for the kernel that clears them
    w.x = p; p += T * m.d; w.q = p; p += T * qd; w.k = p; p += T * kd; w.v = p; p += T * kd; w.g = p; p += T * m.dff; w.u = p; p += T * m.dff;
    w.qn = p; p += T * qd; w.att = p; p += T * qd; w.kn = p;
    return true;
}
void free_work(Work &w) { if (w.base) cudaFree(w.base); w = Work(); }

// products of the same rows with up to three matrices behind the kernel that writes their planes; one launch where their scales
// have one width
struct Product { long long h; int64_t *out; const int64_t *add = nullptr; };
template <typename Write>
bool products(Write write, std::initializer_list<Product> list, const int8_t *planes, long long T, long long frac, const int64_t *in, long long in_n) {
    Q1Part parts[Q1_MAX_PARTS];
    int n = 0;
    bool sc32 = true, same = true;
    for (const Product &p : list) {
        const Q1Weight &w = q_w[(size_t)p.h];
        same = same && (n == 0 || w.sc32 == sc32);
        sc32 = w.sc32;
        parts[n++] = {w.units, w.out_f, p.out, p.add, w.max_scale};
    }
    const long long nb = q_w[(size_t)list.begin()->h].nb;
    if (same) return planes_and_products(write, parts, n, sc32, nb, planes, T, frac, in, nullptr, in_n, q_stream);
    for (int i = 0; i < n; i++)
        if (!planes_and_products(write, parts + i, 1, q_w[(size_t)list.begin()[i].h].sc32, nb, planes, T, frac, in, nullptr, in_n, q_stream)) return false;
    return true;
}
// the same for one row
bool products_of_row(const Q1RowInput &in, std::initializer_list<Product> list, bool swiglu, long long frac) {
    Q1Part parts[Q1_MAX_PARTS];
    int n = 0;
    bool sc32 = true, same = true;
    for (const Product &p : list) {
        const Q1Weight &w = q_w[(size_t)p.h];
        same = same && (n == 0 || w.sc32 == sc32);
        sc32 = w.sc32;
        parts[n++] = {w.units, w.out_f, p.out, p.add, w.max_scale};
    }
    const long long nb = q_w[(size_t)list.begin()->h].nb;
    if (swiglu && same && nb <= 32) return row_products(parts, n, sc32, nb, in, true, frac, q_stream);
    if (same) { if (!row_products(parts, n, sc32, nb, in, false, frac, q_stream)) return false; }
    else
        for (int i = 0; i < n; i++)
            if (!row_products(parts + i, 1, q_w[(size_t)list.begin()[i].h].sc32, nb, in, false, frac, q_stream)) return false;
    return !swiglu || launch_q1_silu_mul(parts[0].out, parts[1].out, parts[0].out_f, (int)frac, parts[0].out, q_stream) == cudaSuccess;
}

// the per-head norms: w.q, w.k -> w.qn, w.kn
bool head_norms(const Q1Stack &m, size_t layer, Work &w, long long T, int *flags) {
    const int f = (int)m.frac;
    return launch_rmsnorm(w.q, T * m.H, m.hd, q_bufs[(size_t)m.qng[layer]].p, f, m.eps, w.qn, flags, q_stream) == cudaSuccess &&
           launch_rmsnorm(w.k, T * m.Hkv, m.hd, q_bufs[(size_t)m.kng[layer]].p, f, m.eps, w.kn, flags, q_stream) == cudaSuccess;
}

// One layer on T rows of w.x.  attend(layer) runs the per-head norms of w.q and w.k, rotation, cache append and attention into w.att.
template <typename Attend>
bool layer_rows(const Q1Stack &m, long long li, Work &w, long long T, int *flags, Attend attend) {
    const size_t i = (size_t)li;
    const long long qd = m.H * m.hd, widest = std::max({m.d, qd, m.dff});
    const int f = (int)m.frac;
    int8_t *planes = T > 1 ? (int8_t *)q_ensure(QR_PLANES, (size_t)T * 8 * (size_t)widest) : nullptr;
    if (T > 1 && !planes) return false;
    auto gain = [&](long long h) { return q_bufs[(size_t)h].p; };
    auto norm = [&](long long h) {
        return [&, h](const PlaneDuties &d) { return launch_rmsnorm_planes(w.x, T, m.d, gain(h), f, m.eps, nullptr, planes, flags, d, q_stream); };
    };
    bool ok = (T == 1 ? products_of_row({w.x, true, gain(m.n1g[i]), m.eps, true}, {{m.wq[i], w.q}, {m.wk[i], w.k}, {m.wv[i], w.v}}, false, m.frac)
                      : products(norm(m.n1g[i]), {{m.wq[i], w.q}, {m.wk[i], w.k}, {m.wv[i], w.v}}, planes, T, m.frac, w.x, T * m.d)) &&
              attend(i);
    if (T == 1)
        return ok && products_of_row({w.att, false, nullptr, 0}, {{m.wo[i], w.x, w.x}}, false, m.frac) &&
               products_of_row({w.x, true, gain(m.n2g[i]), m.eps, true}, {{m.w1[i], w.g}, {m.wu[i], w.u}}, true, m.frac) &&
               products_of_row({w.g, false, nullptr, 0}, {{m.w2[i], w.x, w.x}}, false, m.frac);
    return ok && products([&](const PlaneDuties &d) { return launch_q1_prep(w.att, T, qd / 128, planes, d, q_stream); },
                          {{m.wo[i], w.x, w.x}}, planes, T, m.frac, w.att, T * qd) &&
           products(norm(m.n2g[i]), {{m.w1[i], w.g}, {m.wu[i], w.u}}, planes, T, m.frac, w.x, T * m.d) &&
           products([&](const PlaneDuties &d) { return launch_q1_prep_swiglu(w.g, w.u, m.dff, f, T, m.dff / 128, planes, d, q_stream); },
                    {{m.w2[i], w.x, w.x}}, planes, T, m.frac, w.g, 2 * T * m.dff);
}

// logits of `rows` rows starting at x: final norm, output matrix
bool head_rows(const Q1Stack &m, const int64_t *x, long long rows, int64_t *logits, int *flags) {
    const int64_t *gain = q_bufs[(size_t)m.finalg].p;
    if (rows == 1) return products_of_row({x, true, gain, m.eps, true}, {{m.out_head, logits}}, false, m.frac);
    int8_t *planes = (int8_t *)q_ensure(QR_PLANES, (size_t)rows * 8 * (size_t)m.d);
    if (!planes) return false;
    return products([&](const PlaneDuties &d) { return launch_rmsnorm_planes(x, rows, m.d, gain, (int)m.frac, m.eps, nullptr, planes, flags, d, q_stream); },
                    {{m.out_head, logits}}, planes, rows, m.frac, x, rows * m.d);
}

// The same for a step's rows, the output matrix in two halves of whole waves where it is large: the first half's logits are on their way to
// the host while the second is multiplied (7 MB take 130 us, the product of six rows 120), as long as nothing was refused: behind the first
// half the flags say all that they will but whether a wait of the second product gave up.  No tile of either half is split among CTAs
// (q1_tc_split), which up to 64 tokens takes four waves of tiles each: a matrix of fewer than 151552 rows is one piece (a step of two layers and
// six sequences 457 us with 151936 rows in halves, 464 with 128256 in one piece).  `first`: rows of the first half, 0 for one piece; its logits
// [rows][first] lie in front of the others'.
cudaStream_t q_copy = nullptr;
cudaEvent_t q_half = nullptr;
long long head_first(const Q1Stack &m, long long rows) {
    const Q1Weight &w = q_w[(size_t)m.out_head];
    const long long tiles = (w.out_f + 127) / 128, first = tiles / 2 / Q1_TC_CTAS * Q1_TC_CTAS;
    if (rows < 2 || first <= 0 || q1_tc_split(first, rows) || q1_tc_split(tiles - first, rows)) return 0;
    if (!q_copy && cudaStreamCreateWithFlags(&q_copy, cudaStreamNonBlocking) != cudaSuccess) { cudaGetLastError(); q_copy = nullptr; return 0; }
    if (!q_half && cudaEventCreateWithFlags(&q_half, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); q_half = nullptr; return 0; }
    return first * 128;
}
bool head_halves(const Q1Stack &m, const int64_t *x, long long rows, long long first, int64_t *logits, int *flags) {
    const Q1Weight &w = q_w[(size_t)m.out_head];
    int8_t *planes = (int8_t *)q_ensure(QR_PLANES, (size_t)rows * 8 * (size_t)m.d);
    const PlaneDuties d = next_digits(q_stream);
    const Q1Part a = {w.units, first, logits, nullptr, w.max_scale},
                 b = {w.units + (size_t)(first / 16) * w.nb * q1_unit_bytes(w.sc32), w.out_f - first, logits + rows * first, nullptr, w.max_scale};
    return planes && d.nl &&
           launch_rmsnorm_planes(x, rows, m.d, q_bufs[(size_t)m.finalg].p, (int)m.frac, m.eps, nullptr, planes, flags, d, q_stream) == cudaSuccess &&
           launch_q1_apply(&a, 1, w.sc32, w.nb, planes, rows, m.frac, d.nl, q_stream) == cudaSuccess && cudaEventRecord(q_half, q_stream) == cudaSuccess &&
           launch_q1_apply(&b, 1, w.sc32, w.nb, planes, rows, m.frac, d.nl, q_stream) == cudaSuccess;
}
bool copy_half(long long *out, const int64_t *logits, long long rows, long long vocab, long long from, long long n, cudaStream_t s) {
    return cudaMemcpy2DAsync(out + from, (size_t)vocab * 8, logits + rows * from, (size_t)n * 8, (size_t)n * 8, (size_t)rows, cudaMemcpyDeviceToHost, s) == cudaSuccess;
}

// Rows from pageable host memory: four threads copy pieces into a page-locked buffer and send each on its way (one thread, or the
// driver's own staging, copies 11 GB/s: 1.4 ms for 512 rows of 4096).  A single buffer of at most 32 MB, kept until the
// weights are freed.
uint8_t *q_pin = nullptr;
size_t q_pin_cap = 0;
void free_pin() {
    if (q_pin) cudaFreeHost(q_pin);
    if (q_stage) cudaFreeHost(q_stage);
    q_pin = q_stage = nullptr;
    q_pin_cap = 0; q_stage_tried = false;
}
bool upload_rows(int64_t *dst, const long long *src, size_t bytes) {
    constexpr size_t LEAST = 1 << 20, MOST = 32 << 20, PIECE = 512 << 10;
    constexpr int THREADS = 4;
    uint8_t *&pin = q_pin;
    size_t &cap = q_pin_cap;
    if (bytes < LEAST) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    const size_t want = std::min(bytes, MOST);
    if (cap < want) {
        if (pin) { cudaStreamSynchronize(q_stream); free_pin(); }
        if (cudaHostAlloc(&pin, want, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError(); pin = nullptr;
            return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
        }
        cap = want;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    for (size_t part = 0; part < bytes; part += cap) {
        const size_t n = std::min(cap, bytes - part), pieces = (n + PIECE - 1) / PIECE;
        if (part && cudaStreamSynchronize(q_stream) != cudaSuccess) return false;
        std::atomic<size_t> next{0};
        std::atomic<bool> good{true};
        auto copy = [&]() {
            if (cudaSetDevice(dev) != cudaSuccess) { good = false; return; }
            for (size_t i; (i = next.fetch_add(1)) < pieces;) {
                const size_t at = i * PIECE, len = std::min(PIECE, n - at);
                memcpy(pin + at, (const uint8_t *)src + part + at, len);
                if (cudaMemcpyAsync((uint8_t *)dst + part + at, pin + at, len, cudaMemcpyHostToDevice, q_stream) != cudaSuccess) good = false;
            }
        };
        run_with_helpers<THREADS - 1>(copy);
        if (!good) return false;
    }
    return true;
}

// int64 host rows -> int32; false when a value does not fit
bool narrow(const long long *src, size_t n, std::vector<int32_t> &dst) {
    dst.resize(n);
    bool fits = true;
    for (size_t i = 0; i < n; i++) {
        fits = fits && src[i] >= INT32_MIN && src[i] <= INT32_MAX;
        dst[i] = (int32_t)src[i];
    }
    return fits;
}

// `rows` rows of `hd` int64 values -> int32 rows of `hp` >= hd values (zero-filled); false when a value does not fit
bool narrow_rows(const long long *src, size_t rows, long long hd, long long hp, std::vector<int32_t> &dst) {
    dst.assign(rows * (size_t)hp, 0);
    bool fits = true;
    for (size_t r = 0; r < rows; r++)
        for (long long e = 0; e < hd; e++) {
            const long long x = src[r * (size_t)hd + (size_t)e];
            fits = fits && x >= INT32_MIN && x <= INT32_MAX;
            dst[r * (size_t)hp + (size_t)e] = (int32_t)x;
        }
    return fits;
}

// smallest head width the attention kernels take that holds `hd` columns (0: none)
long long padded_head_dim(long long hd) {
    for (long long w : {32LL, 64LL, 128LL, 256LL}) if (hd <= w) return w;
    return 0;
}

// The flags of one of these host calls are a word of its own: the shared word is read and cleared by other threads' calls, whose flags it
// holds meanwhile.  Cleared and read on the stream, one wait.
struct FlagScope {
    int *const word = q_cells + 4, *const before;
    bool ok = false;
    FlagScope() : before(iie::set_flag_word(word)) { ok = cudaMemsetAsync(word, 0, sizeof(int), q_stream) == cudaSuccess; }
    ~FlagScope() { iie::set_flag_word(before); }
    FlagScope(const FlagScope &) = delete;
    FlagScope &operator=(const FlagScope &) = delete;
    int read(cudaStream_t s) const {                   // negative on a CUDA failure
        int pageable = 0, *seen = staging() ? reinterpret_cast<int *>(q_stage) : &pageable;
        if (!ok || cudaMemcpyAsync(seen, word, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return -1;
        return *seen;
    }
    int finish() const { return read(q_stream); }
};

struct DecodeCtx {
    bool alive = false;
    Q1Stack m;
    long long B = 0, cap = 0, vocab = 0;
    int32_t *K = nullptr, *V = nullptr;            // [n_layers][B][Hkv][cap][hd]
    int64_t *logits = nullptr;
    int *pos = nullptr;                            // [B]: where the sequences stand in the step under way
    std::vector<int> at;                           // the same on the host
    Work w;
    std::vector<char> wide;                        // per sequence: a seeded value did not fit the int32 rows
};
std::vector<DecodeCtx> q_ctx;
bool valid_ctx(long long h) { return h >= 0 && (size_t)h < q_ctx.size() && q_ctx[(size_t)h].alive; }
void free_ctx(DecodeCtx &c) {
    if (c.K) cudaFree(c.K);
    if (c.V) cudaFree(c.V);
    if (c.logits) cudaFree(c.logits);
    if (c.pos) cudaFree(c.pos);
    free_work(c.w);
    c = DecodeCtx();
}

}  // namespace

extern "C" long long bonsai_buf_upload_i64(const long long *host, long long n) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!host || n <= 0 || !q_init()) return -1;
    DevBuf b;
    if (cudaMalloc(&b.p, (size_t)n * 8) != cudaSuccess) { cudaGetLastError(); return -1; }
    if (cudaMemcpy(b.p, host, (size_t)n * 8, cudaMemcpyHostToDevice) != cudaSuccess) { cudaGetLastError(); cudaFree(b.p); return -1; }
    b.n = (size_t)n;
    q_bufs.push_back(b);
    return (long long)q_bufs.size() - 1;
}

extern "C" int bonsai_attention_prefill_gpu(const long long *q, const long long *k, const long long *v, long long H, long long Hkv,
                                            long long hd, long long M, long long L, long long start, long long frac,
                                            long long inv_sqrt_fp, long long *out) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    const long long hp = padded_head_dim(hd);          // zero columns change neither a score nor a kept output column
    if (!q || !k || !v || !out || H <= 0 || Hkv <= 0 || hd <= 0 || M <= 0 || L <= 0 || start < 0 || frac < 1 || frac > 29 || H % Hkv ||
        L != start + M || hp == 0 || !attn_shape_ok((int)H, (int)Hkv, (int)hp)) return fail(1, "prefill attention: bad arguments");
    if (!q_init()) return fail(1, "prefill attention: no usable CUDA device");
    // this library's layouts: queries and new K/V rows token-major, the cache [Hkv][L][hp] int32
    const size_t qd = (size_t)(H * hp), kd = (size_t)(Hkv * hp);
    std::vector<int64_t> qt((size_t)M * qd, 0), kt((size_t)M * kd, 0), vt((size_t)M * kd, 0);
    for (long long h = 0; h < H; h++) for (long long t = 0; t < M; t++)
        memcpy(&qt[(size_t)t * qd + (size_t)(h * hp)], q + ((size_t)h * M + t) * hd, (size_t)hd * 8);
    for (long long h = 0; h < Hkv; h++) for (long long t = 0; t < M; t++) {
        memcpy(&kt[(size_t)t * kd + (size_t)(h * hp)], k + ((size_t)h * L + start + t) * hd, (size_t)hd * 8);
        memcpy(&vt[(size_t)t * kd + (size_t)(h * hp)], v + ((size_t)h * L + start + t) * hd, (size_t)hd * 8);
    }
    std::vector<int32_t> kc, vc;
    const bool k_fits = narrow_rows(k, (size_t)Hkv * L, hd, hp, kc), v_fits = narrow_rows(v, (size_t)Hkv * L, hd, hp, vc);
    if (!k_fits || !v_fits) return fail(2, "prefill attention: a K/V value is beyond int32");
    int64_t *dq = nullptr, *dk = nullptr, *dv = nullptr, *dout = nullptr; int32_t *dkc = nullptr, *dvc = nullptr;
    bool ok = cudaMalloc(&dq, qt.size() * 8) == cudaSuccess && cudaMalloc(&dk, kt.size() * 8) == cudaSuccess &&
              cudaMalloc(&dv, vt.size() * 8) == cudaSuccess && cudaMalloc(&dout, qt.size() * 8) == cudaSuccess &&
              cudaMalloc(&dkc, kc.size() * 4) == cudaSuccess && cudaMalloc(&dvc, vc.size() * 4) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(dq, qt.data(), qt.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dk, kt.data(), kt.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dv, vt.data(), vt.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dkc, kc.data(), kc.size() * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dvc, vc.data(), vc.size() * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    int flags = -1;
    if (ok) {
        FlagScope scope;
        ok = scope.ok && iie_attn_prefill_dev(dq, dk, dv, dkc, dvc, start, M, 0, nullptr, nullptr, 0, (int)H, (int)Hkv, (int)hp, L, (int)frac,
                                              inv_sqrt_fp, dout, q_stream) == 0;
        flags = scope.finish();
        ok = ok && flags >= 0 && !(flags & FLAG_GAVE_UP);
    }
    if (ok && flags == 0) {
        ok = cudaMemcpy(qt.data(), dout, qt.size() * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
        if (ok) for (long long h = 0; h < H; h++) for (long long t = 0; t < M; t++)
            memcpy(out + ((size_t)h * M + t) * hd, &qt[(size_t)t * qd + (size_t)(h * hp)], (size_t)hd * 8);
    }
    for (void *p : {(void *)dq, (void *)dk, (void *)dv, (void *)dout, (void *)dkc, (void *)dvc}) if (p) cudaFree(p);
    if (!ok) return fail(1, "prefill attention: CUDA failure");
    if (flags) return fail(2, "prefill attention: a value left the exact envelope");
    return 0;
}

extern "C" int bonsai_attention_decode_batched_gpu(const long long *q, const long long *Kc, const long long *Vc, const long long *lengths,
                                                   long long B, long long H, long long Hkv, long long hd, long long cap, long long frac,
                                                   long long inv_sqrt_fp, long long *out) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    const long long hp = padded_head_dim(hd);
    if (!q || !Kc || !Vc || !lengths || !out || B <= 0 || H <= 0 || Hkv <= 0 || hd <= 0 || cap <= 0 || H % Hkv || frac < 1 || frac > 29 ||
        hp == 0 || !attn_shape_ok((int)H, (int)Hkv, (int)hp)) return fail(1, "batched decode attention: bad arguments");
    for (long long b = 0; b < B; b++) if (lengths[b] < 1 || lengths[b] > cap) return fail(1, "batched decode attention: a length is outside 1..cap");
    if (!q_init()) return fail(1, "batched decode attention: no usable CUDA device");
    const size_t qd = (size_t)(H * hp), kd = (size_t)(Hkv * hp), per_src = (size_t)Hkv * cap * hd, per = (size_t)Hkv * cap * hp;
    std::vector<int32_t> kc, vc;
    const bool k_fits = narrow_rows(Kc, (size_t)B * Hkv * cap, hd, hp, kc), v_fits = narrow_rows(Vc, (size_t)B * Hkv * cap, hd, hp, vc);
    if (!k_fits || !v_fits) {
        // padding rows beyond a sequence's length are not attended to: only values inside the lengths count
        bool fits = true;
        for (long long b = 0; b < B && fits; b++) for (long long h = 0; h < Hkv && fits; h++)
            for (size_t i = 0; i < (size_t)lengths[b] * hd; i++) {
                const size_t at = (size_t)b * per_src + (size_t)h * cap * hd + i;
                if (Kc[at] < INT32_MIN || Kc[at] > INT32_MAX || Vc[at] < INT32_MIN || Vc[at] > INT32_MAX) { fits = false; break; }
            }
        if (!fits) return fail(2, "batched decode attention: a K/V value is beyond int32");
    }
    // the newest row of every sequence (position length - 1) is passed as the step's K/V row and rewritten unchanged
    std::vector<int64_t> qp((size_t)B * qd, 0), kn((size_t)B * kd, 0), vn((size_t)B * kd, 0);
    for (long long b = 0; b < B; b++) {
        for (long long h = 0; h < H; h++) memcpy(&qp[(size_t)b * qd + (size_t)(h * hp)], q + ((size_t)b * H + h) * hd, (size_t)hd * 8);
        for (long long h = 0; h < Hkv; h++) {
            const size_t src = (size_t)b * per_src + ((size_t)h * cap + (size_t)(lengths[b] - 1)) * hd;
            memcpy(&kn[(size_t)b * kd + (size_t)(h * hp)], Kc + src, (size_t)hd * 8);
            memcpy(&vn[(size_t)b * kd + (size_t)(h * hp)], Vc + src, (size_t)hd * 8);
        }
    }
    int64_t *dq = nullptr, *dk = nullptr, *dv = nullptr, *dout = nullptr; int32_t *dkc = nullptr, *dvc = nullptr;
    bool ok = cudaMalloc(&dq, qp.size() * 8) == cudaSuccess && cudaMalloc(&dout, qp.size() * 8) == cudaSuccess &&
              cudaMalloc(&dk, kn.size() * 8) == cudaSuccess && cudaMalloc(&dv, vn.size() * 8) == cudaSuccess &&
              cudaMalloc(&dkc, kc.size() * 4) == cudaSuccess && cudaMalloc(&dvc, vc.size() * 4) == cudaSuccess;
    ok = ok && cudaMemcpyAsync(dq, qp.data(), qp.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dk, kn.data(), kn.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dv, vn.data(), vn.size() * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dkc, kc.data(), kc.size() * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
         cudaMemcpyAsync(dvc, vc.data(), vc.size() * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    int flags = -1;
    if (ok) {
        FlagScope scope;
        ok = scope.ok;
        for (long long b = 0; ok && b < B; b++)
            ok = iie_attn_decode_dev(dq + (size_t)b * qd, dk + (size_t)b * kd, dv + (size_t)b * kd, dkc + (size_t)b * per, dvc + (size_t)b * per,
                                     lengths[b] - 1, nullptr, 0, nullptr, nullptr, 0, (int)H, (int)Hkv, (int)hp, cap, (int)frac, inv_sqrt_fp,
                                     dout + (size_t)b * qd, q_stream) == 0;
        flags = scope.finish();
        ok = ok && flags >= 0 && !(flags & FLAG_GAVE_UP);
    }
    if (ok && flags == 0) {
        ok = cudaMemcpy(qp.data(), dout, qp.size() * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
        if (ok) for (long long b = 0; b < B; b++) for (long long h = 0; h < H; h++)
            memcpy(out + ((size_t)b * H + h) * hd, &qp[(size_t)b * qd + (size_t)(h * hp)], (size_t)hd * 8);
    }
    for (void *p : {(void *)dq, (void *)dk, (void *)dv, (void *)dout, (void *)dkc, (void *)dvc}) if (p) cudaFree(p);
    if (!ok) return fail(1, "batched decode attention: CUDA failure");
    if (flags) return fail(2, "batched decode attention: a value left the exact envelope");
    return 0;
}

extern "C" int bonsai_prefill_forward_gpu(const long long *x_embed, long long T, long long d, long long n_layers, long long H, long long Hkv,
                                          long long hd, long long dff, long long frac, long long eps, long long inv_sqrt_fp,
                                          const long long *wq, const long long *wk, const long long *wv, const long long *wo,
                                          const long long *w1, const long long *wu, const long long *w2, const long long *n1g,
                                          const long long *n2g, const long long *qng, const long long *kng, long long finalg,
                                          long long out_head, long long cos_h, long long sin_h, long long *out_logits, long long *out_k,
                                          long long *out_v) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!x_embed || !out_logits || T <= 0 || T > (1 << 20) || n_layers <= 0 || eps < 0 || !wq || !wk || !wv || !wo || !w1 || !wu || !w2 || !n1g ||
        !n2g || !qng || !kng) return fail(1, "prefill forward: bad arguments");
    if (!q_init()) return fail(1, "prefill forward: no usable CUDA device");
    Q1Stack m;
    m.n_layers = n_layers; m.H = H; m.Hkv = Hkv; m.hd = hd; m.d = d; m.dff = dff; m.frac = frac; m.eps = (unsigned long long)eps;
    m.inv_sqrt = inv_sqrt_fp; m.finalg = finalg; m.out_head = out_head; m.cos_h = cos_h; m.sin_h = sin_h;
    fill_stack(m, wq, wk, wv, wo, w1, wu, w2, n1g, n2g, qng, kng);
    if (!stack_ok(m, T)) return fail(1, "prefill forward: a handle or a dimension does not fit the model");
    const long long vocab = q_w[(size_t)out_head].out_f;
    const size_t kv_elems = (size_t)Hkv * T * hd;
    Work w;
    PromptBuffers buffers;
    int32_t *kc = (int32_t *)q_ensure(QR_KEYS, kv_elems * 4), *vc = (int32_t *)q_ensure(QR_VALUES, kv_elems * 4);
    int64_t *logits = (int64_t *)q_ensure(QR_LOGITS, (size_t)vocab * 8);
    bool ok = kc && vc && logits && alloc_work(w, m, T, true);
    ok = ok && upload_rows(w.x, x_embed, (size_t)T * d * 8);
    int flags = -1;
    std::vector<int32_t> rows;
    if (ok) {
        FlagScope scope;
        ok = scope.ok;
        int *const fw = scope.word;
        const int64_t *cosd = q_bufs[(size_t)cos_h].p, *sind = q_bufs[(size_t)sin_h].p;
        for (long long li = 0; ok && li < n_layers; li++) {
            ok = layer_rows(m, li, w, T, fw, [&](size_t layer) {
                return head_norms(m, layer, w, T, fw) &&
                       iie_attn_prefill_dev(w.qn, w.kn, w.v, kc, vc, 0, T, 0, cosd, sind, 2, (int)H, (int)Hkv, (int)hd, T, (int)frac, inv_sqrt_fp, w.att,
                                            q_stream) == 0;
            });
            if (ok && (out_k || out_v)) {
                // the layer's cache is the export: K after head norm and rotation, V as projected, [Hkv][T][hd]
                rows.resize(kv_elems);
                for (int which = 0; ok && which < 2; which++) {
                    long long *dst = which ? out_v : out_k;
                    if (!dst) continue;
                    ok = cudaMemcpyAsync(rows.data(), which ? vc : kc, kv_elems * 4, cudaMemcpyDeviceToHost, q_stream) == cudaSuccess &&
                         cudaStreamSynchronize(q_stream) == cudaSuccess;
                    if (ok) for (size_t i = 0; i < kv_elems; i++) dst[(size_t)li * kv_elems + i] = rows[i];
                }
            }
        }
        ok = ok && head_rows(m, w.x + (size_t)(T - 1) * d, 1, logits, fw);
        flags = scope.finish();
        ok = ok && flags >= 0 && !(flags & FLAG_GAVE_UP);
    }
    if (ok && flags == 0) ok = cudaMemcpy(out_logits, logits, (size_t)vocab * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
    if (!ok) { cudaStreamSynchronize(q_stream); return fail(1, "prefill forward: CUDA failure"); }
    if (flags) return fail(4, "prefill forward: a value left the exact envelope");
    return 0;
}

extern "C" long long bonsai_decode_ctx_create(long long B, long long n_layers, long long H, long long Hkv, long long hd, long long d,
                                              long long dff, long long cap, long long vocab, long long frac, long long eps,
                                              long long inv_sqrt, const long long *wq, const long long *wk, const long long *wv,
                                              const long long *wo, const long long *w1, const long long *wu, const long long *w2,
                                              const long long *n1g, const long long *n2g, const long long *qng, const long long *kng,
                                              long long finalg, long long out_head, long long cos_h, long long sin_h) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (B <= 0 || B > 4096 || n_layers <= 0 || cap <= 0 || vocab <= 0 || eps < 0 || !wq || !wk || !wv || !wo || !w1 || !wu || !w2 || !n1g || !n2g ||
        !qng || !kng || !q_init()) { fail(1, "decode context: bad arguments"); return -1; }
    DecodeCtx c;
    Q1Stack &m = c.m;
    m.n_layers = n_layers; m.H = H; m.Hkv = Hkv; m.hd = hd; m.d = d; m.dff = dff; m.frac = frac; m.eps = (unsigned long long)eps;
    m.inv_sqrt = inv_sqrt; m.finalg = finalg; m.out_head = out_head; m.cos_h = cos_h; m.sin_h = sin_h;
    fill_stack(m, wq, wk, wv, wo, w1, wu, w2, n1g, n2g, qng, kng);
    if (!stack_ok(m, cap) || q_w[(size_t)out_head].out_f != vocab) { fail(1, "decode context: a handle or a dimension does not fit the model"); return -1; }
    c.B = B; c.cap = cap; c.vocab = vocab; c.wide.assign((size_t)B, 0); c.at.assign((size_t)B, 0);
    const size_t kv = (size_t)n_layers * B * Hkv * cap * hd * 4;
    if (cudaMalloc(&c.K, kv) != cudaSuccess || cudaMalloc(&c.V, kv) != cudaSuccess || cudaMemset(c.K, 0, kv) != cudaSuccess ||
        cudaMemset(c.V, 0, kv) != cudaSuccess || cudaMalloc(&c.logits, (size_t)B * vocab * 8) != cudaSuccess || cudaMalloc(&c.pos, (size_t)B * 4) != cudaSuccess || !alloc_work(c.w, m, B, false)) {
        cudaGetLastError(); free_ctx(c); fail(2, "decode context: out of device memory"); return -1;
    }
    c.alive = true;
    size_t slot = q_ctx.size();
    for (size_t i = 0; i < q_ctx.size(); i++) if (!q_ctx[i].alive) { slot = i; break; }
    if (slot == q_ctx.size()) q_ctx.emplace_back();
    q_ctx[slot] = std::move(c);
    return (long long)slot;
}

extern "C" int bonsai_decode_ctx_seed_seq(long long ctx_h, long long b, const long long *k_src, const long long *v_src, long long Lb) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!valid_ctx(ctx_h)) return fail(1, "decode context: no such context");
    DecodeCtx &c = q_ctx[(size_t)ctx_h];
    if (b < 0 || b >= c.B || Lb < 0 || Lb > c.cap || (Lb > 0 && (!k_src || !v_src))) return fail(1, "decode context: bad sequence or length");
    if (Lb == 0) return 0;
    const Q1Stack &m = c.m;
    const size_t n = (size_t)m.n_layers * m.Hkv * Lb * m.hd;
    std::vector<int32_t> kn, vn;
    const bool fits_k = narrow(k_src, n, kn), fits_v = narrow(v_src, n, vn);
    if (!fits_k || !fits_v) c.wide[(size_t)b] = 1;           // the next step of this context reports the overflow status
    bool ok = true;
    for (long long li = 0; ok && li < m.n_layers; li++) for (long long h = 0; ok && h < m.Hkv; h++) {
        const size_t src = ((size_t)li * m.Hkv + h) * Lb * m.hd, dst = ((((size_t)li * c.B + b) * m.Hkv + h) * c.cap) * m.hd;
        ok = cudaMemcpyAsync(c.K + dst, kn.data() + src, (size_t)Lb * m.hd * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
             cudaMemcpyAsync(c.V + dst, vn.data() + src, (size_t)Lb * m.hd * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    }
    ok = ok && cudaStreamSynchronize(q_stream) == cudaSuccess;
    return ok ? 0 : fail(1, "decode context: CUDA failure");
}

extern "C" int bonsai_decode_step(long long ctx_h, const long long *x_in, const long long *pos, long long *out_logits) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    clear_error();
    if (!valid_ctx(ctx_h) || !x_in || !pos || !out_logits) return fail(1, "decode step: bad arguments");
    DecodeCtx &c = q_ctx[(size_t)ctx_h];
    const Q1Stack &m = c.m;
    for (long long b = 0; b < c.B; b++) if (pos[b] < 0 || pos[b] >= c.cap) return fail(1, "decode step: a position is outside the cache");
    for (char wide : c.wide) if (wide) return fail(4, "decode step: a seeded K/V value is beyond int32");
    const long long qd = m.H * m.hd, kd = m.Hkv * m.hd;
    const size_t per_seq = (size_t)m.Hkv * c.cap * m.hd;
    std::copy(pos, pos + c.B, c.at.begin());
    const long long longest = *std::max_element(pos, pos + c.B);
    bool ok = cudaMemcpyAsync(c.w.x, x_in, (size_t)c.B * m.d * 8, cudaMemcpyHostToDevice, q_stream) == cudaSuccess &&
              cudaMemcpyAsync(c.pos, c.at.data(), (size_t)c.B * 4, cudaMemcpyHostToDevice, q_stream) == cudaSuccess;
    int flags = -1;
    {
        FlagScope scope;
        ok = ok && scope.ok;
        int *const fw = scope.word;
        const int64_t *cosd = q_bufs[(size_t)m.cos_h].p, *sind = q_bufs[(size_t)m.sin_h].p;
        for (long long li = 0; ok && li < m.n_layers; li++) {
            int32_t *Kl = c.K + (size_t)li * c.B * per_seq, *Vl = c.V + (size_t)li * c.B * per_seq;
            ok = layer_rows(m, li, c.w, c.B, fw, [&](size_t layer) {
                // sequences sit at their own positions: one launch for all of them, else one single-token attention per sequence
                const int64_t *qg = q_bufs[(size_t)m.qng[layer]].p, *kg = q_bufs[(size_t)m.kng[layer]].p;
                const int rc = c.B == 1 ? attn_decode_normed(c.w.q, c.w.k, c.w.v, Kl, Vl, pos[0], nullptr, cosd, sind, 2, (int)m.H, (int)m.Hkv, (int)m.hd,
                                                             c.cap, (int)m.frac, m.inv_sqrt, qg, kg, m.eps, c.w.att, q_stream)
                                        : attn_decode_each(c.w.q, c.w.k, c.w.v, Kl, Vl, c.pos, longest, c.B, (long long)per_seq, cosd, sind, 2, (int)m.H,
                                                           (int)m.Hkv, (int)m.hd, c.cap, (int)m.frac, m.inv_sqrt, qg, kg, m.eps, c.w.att, q_stream);
                if (rc != 3) return rc == 0;
                if (!head_norms(m, layer, c.w, c.B, fw)) return false;
                for (long long b = 0; b < c.B; b++)
                    if (iie_attn_decode_dev(c.w.qn + (size_t)b * qd, c.w.kn + (size_t)b * kd, c.w.v + (size_t)b * kd, Kl + (size_t)b * per_seq,
                                            Vl + (size_t)b * per_seq, pos[b], nullptr, 0, cosd, sind, 2, (int)m.H, (int)m.Hkv, (int)m.hd, c.cap,
                                            (int)m.frac, m.inv_sqrt, c.w.att + (size_t)b * qd, q_stream) != 0) return false;
                return true;
            });
        }
        const long long first = ok ? head_first(m, c.B) : 0;
        if (first) {
            ok = head_halves(m, c.w.x, c.B, first, c.logits, fw) && cudaStreamWaitEvent(q_copy, q_half, 0) == cudaSuccess &&
                 (scope.read(q_copy) != 0 || copy_half(out_logits, c.logits, c.B, c.vocab, 0, first, q_copy));
        } else ok = ok && head_rows(m, c.w.x, c.B, c.logits, fw);
        flags = scope.finish();
        ok = ok && flags >= 0 && !(flags & FLAG_GAVE_UP);
        if (ok && flags == 0)
            ok = first ? copy_half(out_logits, c.logits, c.B, c.vocab, first, c.vocab - first, q_copy)
                       : cudaMemcpyAsync(out_logits, c.logits, (size_t)c.B * c.vocab * 8, cudaMemcpyDeviceToHost, q_stream) == cudaSuccess;
        // (nothing is on its way into the caller's array when the call ends, whatever it returns)
        if (cudaStreamSynchronize(first ? q_copy : q_stream) != cudaSuccess) ok = false;
    }
    if (!ok) return fail(1, "decode step: CUDA failure");
    if (flags) return fail(4, "decode step: a value left the exact envelope");
    return 0;
}

extern "C" void bonsai_decode_ctx_free(long long ctx_h) {
    std::lock_guard<std::recursive_mutex> lk(q_mu);
    if (!valid_ctx(ctx_h)) return;
    cudaDeviceSynchronize();
    free_ctx(q_ctx[(size_t)ctx_h]);
}

static void q1_release_model_state() {
    free_pin();
    for (auto &c : q_ctx) if (c.alive) free_ctx(c);
    q_ctx.clear();
    for (auto &b : q_bufs) if (b.p) cudaFree(b.p);
    q_bufs.clear();
}
