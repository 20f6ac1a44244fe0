// Support kernels around the streamed products: weight repack, activation limb planes, the exact
// 128-bit fallback product, routing (top-k + sigmoid), dispatch, RMSNorm and the unfused
// element-wise steps used by the fallback composition.
#include "kernels.h"
#include "layout.cuh"
#include "norm.cuh"

#include <algorithm>

namespace iie {

unsigned long long g_launches = 0;

namespace {

// ---------------------------------------------------------------------------------------------------
// repack / unpack: one thread per raw byte
// ---------------------------------------------------------------------------------------------------
template <bool FORWARD>
__global__ void repack_kernel(const uint8_t *src, uint8_t *dst, long long out_f, long long nb, int qtype,
                              unsigned *maxbits) {
    const int bs = qtype == QT_Q4K ? 144 : 210;
    const long long total = out_f * nb * bs;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long blk_lin = idx / bs;
        const int i = (int)(idx - blk_lin * bs);
        const long long row = blk_lin / nb, blk = blk_lin - row * nb;
        const long long unit = (row >> 3) * nb + blk;
        const int r = (int)(row & 7);
        const long long packed = qtype == QT_Q4K ? unit * HTB_Q4K + q4k_unit_offset(r, i)
                                                 : unit * HTB_Q6K + q6k_unit_offset(r, i);
        if (FORWARD) {
            dst[packed] = src[idx];
            if (maxbits) {                                  // block scale magnitudes (little-endian halves)
                const int dpos = qtype == QT_Q4K ? 0 : 208;
                if (i == dpos) atomicMax(&maxbits[0], ((unsigned)src[idx] | ((unsigned)src[idx + 1] << 8)) & 0x7FFFu);
                if (qtype == QT_Q4K && i == 2)
                    atomicMax(&maxbits[1], ((unsigned)src[idx] | ((unsigned)src[idx + 1] << 8)) & 0x7FFFu);
            }
        } else {
            dst[idx] = src[packed];
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// activation limb planes
// ---------------------------------------------------------------------------------------------------
struct LimbClears { int *a, *b; int64_t *zero; long long zero_n; int8_t *sums; int stride; };      // and sums of 32 columns, see launch_limbs
__device__ __forceinline__ void limb_clears(const LimbClears &c) {
    if (blockIdx.x == 0 && threadIdx.x == 0) { if (c.a) *c.a = 0; if (c.b) *c.b = 0; }
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < c.zero_n; i += (long long)gridDim.x * blockDim.x) c.zero[i] = 0;
}

__global__ void limbs_kernel(const int64_t *x, long long n_rows, long long K, int8_t *planes, int *flags, int *nl_out, const LimbClears clears) {
    pdl_enter();
    limb_clears(clears);
    const long long total = n_rows * K;
    bool bad = false;
    int nl = 0;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long row = idx / K, col = idx - row * K;
        bool ok;
        const uint64_t d = balanced_digits8(x[idx], ok);
        bad |= !ok;
        const int used = d == 0 ? 1 : 8 - (__clzll((long long)d) >> 3);
        nl = used > nl ? used : nl;
#pragma unroll
        for (int l = 0; l < 8; l++) planes[(row * 8 + l) * K + col] = (int8_t)(d >> (8 * l));
    }
    if (bad) atomicOr(flags, 1);
    if (nl_out && nl > 0) atomicMax(nl_out, nl);
}

// The same for K a multiple of 8: a thread takes eight consecutive columns (64 bytes in), transposes the 8 x 8 digit
// bytes in registers and writes eight bytes to each plane.  SUMS: and the sums of 32 columns (a form of its own: rows that need none are
// 0.1 us quicker without their additions, a Q6_K product of 640 x 512 11.6 -> 11.5).
template <bool SUMS>
__global__ void __launch_bounds__(256) limbs8_kernel(const int64_t *x, long long n_rows, long long K, int8_t *planes,
                                                     int *flags, int *nl_out, const LimbClears clears) {
    pdl_enter();
    limb_clears(clears);
    const long long per_row = K >> 3, total = n_rows * per_row;
    bool bad = false;
    uint64_t seen = 0;
    for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total; g += (long long)gridDim.x * blockDim.x) {
        const long long row = g / per_row, col = (g - row * per_row) << 3;
        const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(x + row * K + col);
        uint32_t lo[8], hi[8];
        uint64_t sum_lo = 0;                               // of the low words, and of the signed high words
        int64_t sum_hi = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const ulonglong2 v = __ldcg(src + i);
            if (SUMS) sum_lo += (uint64_t)(uint32_t)v.x + (uint32_t)v.y, sum_hi += (int64_t)(int32_t)(v.x >> 32) + (int32_t)(v.y >> 32);
            bool ok0, ok1;
            const uint64_t d0 = balanced_digits8((int64_t)v.x, ok0), d1 = balanced_digits8((int64_t)v.y, ok1);
            bad |= !ok0 | !ok1;
            seen |= d0 | d1;                               // a digit position is in use if any element has a non-zero digit there or above
            lo[2 * i] = (uint32_t)d0; hi[2 * i] = (uint32_t)(d0 >> 32);
            lo[2 * i + 1] = (uint32_t)d1; hi[2 * i + 1] = (uint32_t)(d1 >> 32);
        }
        int8_t *dst = planes + row * 8 * K + col;
#pragma unroll
        for (int half = 0; half < 2; half++) {             // digits 0..3 from the low words, 4..7 from the high words
            const uint32_t *v = half ? hi : lo;
            uint32_t a[4], b[4];                           // a: elements 0..3, b: elements 4..7, one word per digit
            {
                const uint32_t t0 = __byte_perm(v[0], v[1], 0x5140), t1 = __byte_perm(v[2], v[3], 0x5140);
                const uint32_t t2 = __byte_perm(v[0], v[1], 0x7362), t3 = __byte_perm(v[2], v[3], 0x7362);
                a[0] = __byte_perm(t0, t1, 0x5410); a[1] = __byte_perm(t0, t1, 0x7632);
                a[2] = __byte_perm(t2, t3, 0x5410); a[3] = __byte_perm(t2, t3, 0x7632);
            }
            {
                const uint32_t t0 = __byte_perm(v[4], v[5], 0x5140), t1 = __byte_perm(v[6], v[7], 0x5140);
                const uint32_t t2 = __byte_perm(v[4], v[5], 0x7362), t3 = __byte_perm(v[6], v[7], 0x7362);
                b[0] = __byte_perm(t0, t1, 0x5410); b[1] = __byte_perm(t0, t1, 0x7632);
                b[2] = __byte_perm(t2, t3, 0x5410); b[3] = __byte_perm(t2, t3, 0x7632);
            }
#pragma unroll
            for (int l = 0; l < 4; l++) *reinterpret_cast<uint2 *>(dst + (half * 4 + l) * K) = make_uint2(a[l], b[l]);
        }
        if (SUMS) {                                        // (K is a multiple of 256: four lanes hold the 32 columns of a sub-block)
            for (int off = 1; off <= 2; off <<= 1) { sum_lo += __shfl_xor_sync(0xffffffffu, sum_lo, off); sum_hi += __shfl_xor_sync(0xffffffffu, sum_hi, off); }
            // balanced digits of hi 2^32 + lo: bytes of the sum with 128 added to each of the nine
            const u128 biased = (u128)((i128)sum_hi * ((i128)1 << 32) + (i128)sum_lo) + (((u128)0x80 << 64) | 0x8080808080808080ULL);
            const int t = threadIdx.x & 3;
            const long long j = col >> 5;
            int8_t *to = clears.sums + row * 9 * clears.stride + j;
            for (int l = t; l < 9; l += 4) to[l * clears.stride] = (int8_t)((uint8_t)(biased >> (8 * l)) ^ 0x80);
            for (long long pad = (K >> 5) + t; j == (K >> 5) - 1 && pad < clears.stride; pad += 4)
                for (int l = 0; l < 9; l++) to[l * clears.stride + pad - j] = 0;
        }
    }
    if (bad) atomicOr(flags, 1);
    if (nl_out) {
        // digits in use = position of the highest non-zero digit byte over all elements seen (at least one)
        const int nl = seen == 0 ? 1 : 8 - (__clzll((long long)seen) >> 3);
        atomicMax(nl_out, nl);
    }
}

// ---------------------------------------------------------------------------------------------------
// exact fallback: one thread per output, 128-bit accumulation in the reference's per-weight form
// (north-mini-code/tools/nmc_qk_kernel.c:85-120).  Valid for every int64 input.
// ---------------------------------------------------------------------------------------------------
__global__ void exact_linear_kernel(const uint8_t *w, int qtype, long long out_f, long long nb, const int64_t *x,
                                    long long T, int fw, int64_t *out) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= out_f * T) return;
    const long long o = idx % out_f, t = idx / out_f;
    const int64_t *xt = x + t * nb * 256;
    i128 acc = 0;
    for (long long b = 0; b < nb; b++) {
        const int64_t *xb = xt + b * 256;
        auto byte = [&](int i) { return (int)repacked_byte(w, qtype, nb, o, b, i); };
        if (qtype == QT_Q4K) {
            const int64_t dq = half_to_fixed(byte(0) | (byte(1) << 8), fw), dmq = half_to_fixed(byte(2) | (byte(3) << 8), fw);
            for (int j = 0; j < 8; j++) {
                int sc, mn;
                if (j < 4) { sc = byte(4 + j) & 63; mn = byte(8 + j) & 63; }
                else { sc = (byte(8 + j) & 0xF) | ((byte(j) >> 6) << 4); mn = (byte(8 + j) >> 4) | ((byte(4 + j) >> 6) << 4); }
                const int64_t ws = dq * sc, wm = dmq * mn;
                for (int l = 0; l < 32; l++) {
                    const int q = (byte(16 + 32 * (j >> 1) + l) >> ((j & 1) * 4)) & 0xF;
                    acc += (i128)(ws * q - wm) * xb[32 * j + l];
                }
            }
        } else {
            const int64_t dq = half_to_fixed(byte(208) | (byte(209) << 8), fw);
            for (int sb = 0; sb < 16; sb++) {
                const int half = sb >> 3, k = (sb >> 1) & 3, l0 = (sb & 1) * 16;
                const int64_t ws = dq * (int64_t)(int8_t)byte(192 + 8 * half + 2 * k + (sb & 1));
                for (int l = 0; l < 16; l++) {
                    const int ql = byte(64 * half + 32 * (k & 1) + l0 + l), qh = byte(128 + 32 * half + l0 + l);
                    const int q = (((k < 2) ? (ql & 0xF) : (ql >> 4)) | (((qh >> (2 * k)) & 3) << 4)) - 32;
                    acc += (i128)(ws * q) * xb[16 * sb + l];
                }
            }
        }
    }
    out[t * out_f + o] = (int64_t)(acc >> fw);
}

// Dense int64 weights (router / gain matrices registered as int64): exact 128-bit product; the
// reference additionally requires the un-shifted sum to fit int64 (nmc_qk_cuda.cu:615-638), which is
// reported through flags bit 2.
__global__ void exact_dense_kernel(const int64_t *w, long long out_f, long long in_f, const int64_t *x, long long T,
                                   int fw, int64_t *out, int *flags) {
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= out_f * T) return;
    const long long o = warp % out_f, t = warp / out_f;
    i128 acc = 0;
    for (long long i = lane; i < in_f; i += 32) acc += (i128)w[o * in_f + i] * x[t * in_f + i];
    unsigned long long lo = (unsigned long long)acc, hi = (unsigned long long)((u128)acc >> 64);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const unsigned long long lo2 = __shfl_down_sync(0xffffffffu, lo, s), hi2 = __shfl_down_sync(0xffffffffu, hi, s);
        const u128 sum = (((u128)hi << 64) | lo) + (((u128)hi2 << 64) | lo2);
        lo = (unsigned long long)sum; hi = (unsigned long long)(sum >> 64);
    }
    if (lane == 0) {
        const i128 total = (i128)(((u128)hi << 64) | lo);
        if (total > (i128)INT64_MAX || total < (i128)INT64_MIN) { if (flags) atomicOr(flags, 4); out[t * out_f + o] = 0; }
        else out[t * out_f + o] = ((int64_t)total) >> fw;
    }
}

__global__ void silu_mul_kernel(int64_t *a, const int64_t *b, long long n, int fa) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = mul_shift(silu_fixed(a[i], fa), b[i], fa);
}

__global__ void combine_kernel(const int64_t *dn, const int64_t *gates, long long T, int k, long long d_model, int fa,
                               int64_t *out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T * d_model) return;
    const long long t = i / d_model, o = i - t * d_model;
    unsigned long long acc = 0;
    for (int j = 0; j < k; j++) acc += (unsigned long long)mul_shift(dn[(t * k + j) * d_model + o], gates[t * k + j], fa);
    out[i] = (int64_t)acc;
}

// ---------------------------------------------------------------------------------------------------
// top-k with lowest-index tie-break + sigmoid gates (north-mini-code/src/nmc/cohere2.py:162-165,180)
// ---------------------------------------------------------------------------------------------------
__global__ void topk_kernel(const int64_t *logits, long long rows, int n_experts, int k, int fa, int *ids,
                            int64_t *gates) {
    pdl_enter();
    const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const int64_t *lr = logits + row * n_experts;
    unsigned taken = 0;                                   // bit i: element lane + 32*i already selected
    // a round finds the largest high word, among those the largest low word, among those the lowest id (three warp reductions); the gates of 32
    // rounds are computed side by side
    for (int r0 = 0; r0 < k; r0 += 32) {
        int64_t mine = 0; int mine_id = -1;               // of round r0 + lane
        for (int r = r0; r < min(k, r0 + 32); r++) {
            int64_t best = INT64_MIN; int best_id = 0x7fffffff;
            for (int i = 0, e = lane; e < n_experts; i++, e += 32) {
                if (taken & (1u << i)) continue;
                const int64_t v = lr[e];
                if (best_id == 0x7fffffff || v > best) { best = v; best_id = e; }   // ascending e: ties keep the lower id
            }
            const unsigned open = __ballot_sync(0xffffffffu, best_id != 0x7fffffff);
            const bool have = best_id != 0x7fffffff;
            const int hi = __reduce_max_sync(0xffffffffu, have ? (int)(best >> 32) : INT32_MIN);
            const bool at_hi = have && (int)(best >> 32) == hi;
            const unsigned lo = __reduce_max_sync(0xffffffffu, at_hi ? (unsigned)best : 0u);
            const int id = (int)__reduce_min_sync(0xffffffffu, at_hi && (unsigned)best == lo ? (unsigned)best_id : 0x7fffffffu);
            if (open && (id & 31) == lane) taken |= 1u << (id >> 5);
            if (lane == r - r0) { mine = (int64_t)(((uint64_t)(uint32_t)hi << 32) | lo); mine_id = open ? id : -1; }
        }
        if (r0 + lane < k) {
            ids[row * k + r0 + lane] = mine_id;
            gates[row * k + r0 + lane] = mine_id < 0 ? 0 : sigmoid_fixed(mine, fa);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// dispatch: stable counting sort of (token, slot) pairs by expert, single CTA.  Warp w owns the w-th
// contiguous slice of the pair list; inside a slice, 32 pairs at a time are ranked with a warp match,
// so expert e's pairs keep ascending pair index.  Slots whose expert id falls outside
// [expert_base, expert_base + n_experts) are dropped (they belong to another expert shard).
// ---------------------------------------------------------------------------------------------------
__global__ void dispatch_kernel(const int *ids, const int64_t *gates, long long T, int k, int n_experts, int expert_base,
                                int *grp_off, int *pair_tok, int64_t *pair_gate) {
    pdl_enter();
    extern __shared__ int sm[];                           // cnt[nwarps][E], then start[E + 1]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int *cnt = sm, *start = sm + nwarps * n_experts;
    const long long P = T * k;
    const long long per = ((P + nwarps - 1) / nwarps + 31) / 32 * 32;      // slice length, a multiple of 32
    const long long lo = (long long)warp * per, hi = lo + per < P ? lo + per : P;
    for (int i = threadIdx.x; i < nwarps * n_experts; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    int *mine = cnt + warp * n_experts;
    for (long long i0 = lo; i0 < hi; i0 += 32) {
        const long long i = i0 + lane;
        int e = i < hi ? ids[i] - expert_base : -1;
        if (e < 0 || e >= n_experts) e = -1;
        const unsigned m = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && lane == __ffs(m) - 1) mine[e] += __popc(m);
        __syncwarp();
    }
    __syncthreads();
    // per expert: slice counts -> slice offsets inside the expert's range; then the ranges themselves
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) {
        int run = 0;
        for (int w = 0; w < nwarps; w++) { const int c = cnt[w * n_experts + e]; cnt[w * n_experts + e] = run; run += c; }
        start[e] = run;                                  // total of expert e for now
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < n_experts; e++) { const int c = start[e]; start[e] = run; grp_off[e] = run; run += c; }
        start[n_experts] = run; grp_off[n_experts] = run;
    }
    __syncthreads();
    for (long long i0 = lo; i0 < hi; i0 += 32) {
        const long long i = i0 + lane;
        int e = i < hi ? ids[i] - expert_base : -1;
        if (e < 0 || e >= n_experts) e = -1;
        const unsigned m = __match_any_sync(0xffffffffu, e);
        if (e >= 0) {
            const int dst = start[e] + mine[e] + __popc(m & ((1u << lane) - 1));
            pair_tok[dst] = (int)(i / k);
            pair_gate[dst] = gates[i];
        }
        __syncwarp();
        if (e >= 0 && lane == __ffs(m) - 1) mine[e] += __popc(m);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------------
// integer RMSNorm (north-mini-code/src/nmc/_bonsai/fixedpoint.py:32-72), one CTA per row
// ---------------------------------------------------------------------------------------------------
struct NormArgs {
    const int64_t *x;
    long long rows, rows_a;        // rows from rows_a on take gain_b (per-head norms of queries and keys in one launch)
    int width, wpr;                // warps of a row
    bool wide;                     // every row and the gains start on 16 bytes
    const int64_t *gain_a, *gain_b;
    int fa;
    unsigned long long eps;
    int64_t *out;                  // nullable
    int8_t *planes;                // nullable: digit planes [row][8][width]
    int *flags;
    PlaneDuties duties;
};

// The row stays in registers: a thread holds G groups of four consecutive values, a warp 128 values per group, `wpr` warps a row
// (several short rows share a CTA).  One barrier: every warp adds up the warps' sums and takes the root itself.  What bounds it for
// one row is that chain (row load, two rounds of warp reductions, root and reciprocal, quotients: about 4.5 us with the launch; the
// row read twice, a thread taking the root alone and 64-bit quotients for all: 7), for many rows the eight bytes per value in and
// out and the quotients (2048 x 2048: 103 us before).
template <int G>
__global__ void __launch_bounds__(1024) rmsnorm_kernel(const NormArgs a) {
    pdl_enter();
    __shared__ uint64_t s_lo[32], s_hi[32];
    __shared__ uint32_t s_bits[32];
    if (a.duties.nl_clear && blockIdx.x == 0 && threadIdx.x == 0) *a.duties.nl_clear = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < a.duties.zero_n; i += (long long)gridDim.x * blockDim.x) a.duties.zero[i] = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpr = a.wpr, in_row = warp % wpr;      // wpr is 1 or the CTA's warps
    const long long row = wpr == 1 ? (long long)blockIdx.x * (blockDim.x >> 5) + warp : blockIdx.x;
    const bool live = row < a.rows;
    const int64_t *gain = row < a.rows_a ? a.gain_a : a.gain_b;
    const int step = wpr * 128, i0 = in_row * 128 + lane * 4;
    int64_t x[G][4], g[G][4];
    u128 ssq = 0;
    uint64_t mx = 0, gmx = 0;
#pragma unroll
    for (int k = 0; k < G; k++) {
        const bool in = live && i0 + k * step < a.width;
        const int64_t *src = a.x + row * a.width + i0 + k * step, *gs = gain + i0 + k * step;
        longlong2 v0 = make_longlong2(0, 0), v1 = v0, g0 = make_longlong2(1, 1), g1 = g0;
        if (in && a.wide) {
            v0 = *reinterpret_cast<const longlong2 *>(src); v1 = *reinterpret_cast<const longlong2 *>(src + 2);
            if (gain) { g0 = *reinterpret_cast<const longlong2 *>(gs); g1 = *reinterpret_cast<const longlong2 *>(gs + 2); }
        } else if (in) {
            v0 = make_longlong2(src[0], src[1]); v1 = make_longlong2(src[2], src[3]);
            if (gain) { g0 = make_longlong2(gs[0], gs[1]); g1 = make_longlong2(gs[2], gs[3]); }
        }
        x[k][0] = v0.x; x[k][1] = v0.y; x[k][2] = v1.x; x[k][3] = v1.y;
        g[k][0] = g0.x; g[k][1] = g0.y; g[k][2] = g1.x; g[k][3] = g1.y;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint64_t m = uabs64(x[k][e]), gm = uabs64(g[k][e]);
            if ((m >> 32) == 0) ssq += (uint64_t)(uint32_t)m * (uint32_t)m; else ssq += (u128)m * m;
            mx = m > mx ? m : mx; gmx = gm > gmx ? gm : gmx;
        }
    }
    // bit lengths of the largest |x| and |gain|; beyond 2^57 in |x| the sum of squares may wrap and the row is refused
    uint32_t bits = (uint32_t)(64 - __clzll((long long)mx)) | (uint32_t)(64 - __clzll((long long)gmx)) << 8;
    bool beyond = mx > (1ULL << 57);
    uint32_t xb = __reduce_max_sync(0xffffffffu, (bits & 0xFF) | (beyond ? 128u : 0u)), gb = __reduce_max_sync(0xffffffffu, bits >> 8);
    ssq = warp_sum128(ssq);
    if (wpr > 1) {
        if (lane == 0) { s_lo[warp] = (uint64_t)ssq; s_hi[warp] = (uint64_t)(ssq >> 64); s_bits[warp] = xb | gb << 8; }
        __syncthreads();
        ssq = lane < wpr ? ((u128)s_hi[lane] << 64) | s_lo[lane] : (u128)0;
        bits = lane < wpr ? s_bits[lane] : 0;
        ssq = warp_sum128(ssq);
        xb = __reduce_max_sync(0xffffffffu, bits & 0xFF); gb = __reduce_max_sync(0xffffffffu, bits >> 8);
    }
    beyond = (xb & 128u) != 0; xb &= 127u;
    const NormRow nr(ssq, (int)xb, (int)gb, beyond, a.width, a.eps, a.fa, gain != nullptr);
    if (nr.refused) {                                              // nothing is written
        if (live && lane == 0 && in_row == 0) atomicOr(a.flags, 2);
        return;
    }
    const bool fast = nr.fast;
    const uint64_t inv = !fast && nr.rms < (1ULL << 62) ? recip_below(nr.rms) : 0;
    uint64_t gm = 0;                                               // the general form refuses against the row's largest |gain|
    if (!fast && gain) {
        gm = warp_max64(gmx);
        if (wpr > 1) {                                             // (every warp of the CTA is here: a row has one form)
            __shared__ uint64_t s_gm[32];
            if (lane == 0) s_gm[warp] = gm;
            __syncthreads();
            gm = warp_max64(lane < wpr ? s_gm[lane] : 0);
        }
    }
    bool bad = false;
    int nl = 0;
#pragma unroll
    for (int k = 0; k < G; k++) {
        const int i = i0 + k * step;
        const bool in = live && i < a.width;
        int64_t y[4];
        if (fast) {
#pragma unroll
            for (int e = 0; e < 4; e++) y[e] = nr.fast_value((int)x[k][e], (int)g[k][e]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) y[e] = in ? norm_value(x[k][e], nr.rms, inv, gm, g[k][e], gain != nullptr, a.fa, bad) : 0;
        }
        if (in && a.out) {
            int64_t *to = a.out + row * a.width + i;
            if (a.wide) {
                *reinterpret_cast<longlong2 *>(to) = make_longlong2(y[0], y[1]); *reinterpret_cast<longlong2 *>(to + 2) = make_longlong2(y[2], y[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) to[e] = y[e];
            }
        }
        if (a.planes) {
            uint32_t pl[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (fast) {                                            // byte l of (y + 0x80808080) ^ 0x80808080 is the balanced digit l
                uint32_t d[4];
#pragma unroll
                for (int e = 0; e < 4; e++) d[e] = ((uint32_t)(int)y[e] + 0x80808080u) ^ 0x80808080u;
                const uint32_t any = d[0] | d[1] | d[2] | d[3];
                nl = max(nl, any == 0 ? 1 : 4 - (__clz((int)any) >> 3));
                const uint32_t t0 = __byte_perm(d[0], d[1], 0x5140), t1 = __byte_perm(d[2], d[3], 0x5140);
                const uint32_t t2 = __byte_perm(d[0], d[1], 0x7362), t3 = __byte_perm(d[2], d[3], 0x7362);
                pl[0] = __byte_perm(t0, t1, 0x5410); pl[1] = __byte_perm(t0, t1, 0x7632); pl[2] = __byte_perm(t2, t3, 0x5410); pl[3] = __byte_perm(t2, t3, 0x7632);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    bool ok;
                    const uint64_t d = balanced_digits8(y[e], ok);
                    nl = max(nl, ok ? digits_used(d) : 9);
#pragma unroll
                    for (int l = 0; l < 8; l++) pl[l] |= (uint32_t)((d >> (8 * l)) & 0xFF) << (8 * e);
                }
            }
            if (in) {
#pragma unroll
                for (int l = 0; l < 8; l++) *reinterpret_cast<uint32_t *>(a.planes + (row * 8 + l) * a.width + i) = pl[l];
            }
        }
    }
    if (a.planes && a.duties.nl) {
        nl = __reduce_max_sync(0xffffffffu, live ? nl : 0);
        if (lane == 0 && nl > *(volatile int *)a.duties.nl) atomicMax(a.duties.nl, nl);
    }
    if (live && bad) atomicOr(a.flags, 2);
}

// any width: one CTA per row, values read again for the quotients
__global__ void __launch_bounds__(256) rmsnorm_any_kernel(const NormArgs a) {
    pdl_enter();
    __shared__ uint64_t s_lo[8], s_hi[8], s_max[8], s_gmax[8];
    const long long row = blockIdx.x;
    const int64_t *gain = row < a.rows_a ? a.gain_a : a.gain_b, *xr = a.x + row * a.width;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    u128 ssq = 0;
    uint64_t mx = 0, gm = 0;
    for (int i = tid; i < a.width; i += 256) {
        const uint64_t m = uabs64(xr[i]), gv = gain ? uabs64(gain[i]) : 0;
        ssq += (u128)m * m;
        mx = m > mx ? m : mx; gm = gv > gm ? gv : gm;
    }
    ssq = warp_sum128(ssq); mx = warp_max64(mx); gm = warp_max64(gm);
    if (lane == 0) { s_lo[warp] = (uint64_t)ssq; s_hi[warp] = (uint64_t)(ssq >> 64); s_max[warp] = mx; s_gmax[warp] = gm; }
    __syncthreads();
    ssq = warp_sum128(lane < 8 ? ((u128)s_hi[lane] << 64) | s_lo[lane] : (u128)0);
    mx = warp_max64(lane < 8 ? s_max[lane] : 0); gm = warp_max64(lane < 8 ? s_gmax[lane] : 0);
    const u128 root = isqrt128(ssq / (u128)(unsigned)a.width + a.eps);
    if (mx > (1ULL << 57) || a.width > 8192 || root == 0 || (root >> 64) != 0) { if (tid == 0) atomicOr(a.flags, 2); return; }
    const uint64_t rms = (uint64_t)root, inv = rms < (1ULL << 62) ? recip_below(rms) : 0;
    bool bad = false;
    for (int i = tid; i < a.width; i += 256) a.out[row * a.width + i] = norm_value(xr[i], rms, inv, gm, gain ? gain[i] : 0, gain != nullptr, a.fa, bad);
    if (bad) atomicOr(a.flags, 2);
}

cudaError_t launch_norm(NormArgs a, cudaStream_t s) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.gain_a) | reinterpret_cast<uintptr_t>(a.gain_b) | reinterpret_cast<uintptr_t>(a.out);
    a.wide = (at & 15) == 0;
    if (a.width > 8192 || a.width % 4) {                           // (beyond 8192 every row is refused)
        launch_behind(rmsnorm_any_kernel, (unsigned)a.rows, 256, 0, s, a);
    } else {
        const int groups = (a.width + 127) / 128;                  // of 128 values
        a.wpr = groups <= 2 ? 1 : groups <= 32 ? groups : (groups + 1) / 2;          // one or two groups: a warp per row, eight rows per CTA
        const int threads = a.wpr == 1 ? 256 : a.wpr * 32;
        long long grid = a.wpr == 1 ? (a.rows + 7) / 8 : a.rows;
        grid = std::max(grid, std::min(148LL, a.duties.zero_n / (threads * 8)));     // few rows: more CTAs for the words to clear
        if (groups == 1 || (groups > 2 && groups <= 32)) launch_behind(rmsnorm_kernel<1>, (unsigned)grid, threads, 0, s, a);
        else launch_behind(rmsnorm_kernel<2>, (unsigned)grid, threads, 0, s, a);
    }
    note_launch();
    return cudaGetLastError();
}

inline unsigned grid_for(long long n, int tpb, long long cap = 148LL * 64) {
    long long g = (n + tpb - 1) / tpb;
    if (g > cap) g = cap;
    return (unsigned)(g < 1 ? 1 : g);
}

}  // namespace

cudaError_t launch_repack(const uint8_t *raw, uint8_t *dst, long long out_f, long long nb, int qtype,
                          unsigned *maxbits, cudaStream_t s) {
    const long long total = out_f * nb * (qtype == QT_Q4K ? 144 : 210);
    repack_kernel<true><<<grid_for(total, 256), 256, 0, s>>>(raw, dst, out_f, nb, qtype, maxbits);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_unpack(const uint8_t *src, uint8_t *raw, long long out_f, long long nb, int qtype, cudaStream_t s) {
    const long long total = out_f * nb * (qtype == QT_Q4K ? 144 : 210);
    repack_kernel<false><<<grid_for(total, 256), 256, 0, s>>>(src, raw, out_f, nb, qtype, nullptr);
    note_launch();
    return cudaGetLastError();
}

__global__ void set2_kernel(int *p, int a, int b) {
    pdl_enter();
    p[0] = a; p[1] = b;
}

cudaError_t launch_set2(int *p, int a, int b, cudaStream_t s) {
    launch_behind(set2_kernel, 1, 1, 0, s, p, a, b);
    note_launch();
    return cudaGetLastError();
}

// Selected experts without a binding, compacted in routing order: cold[0] = how many, cold[1..] = their ids
// (north-mini-code/tools/nmc_qk_cuda.cu cold_routes_k).  An id outside the table raises flag bit 1.
__global__ void cold_routes_kernel(const int *ids, int k, const unsigned char *bound, int n_experts, int *cold, int *flags) {
    int n = 0;
    for (int i = 0; i < k; i++) {
        const int e = ids[i];
        if (e < 0 || e >= n_experts) { atomicOr(flags, 2); continue; }
        if (!bound[e]) cold[1 + n++] = e;
    }
    cold[0] = n;
}

cudaError_t launch_cold_routes(const int *ids, int k, const unsigned char *bound, int n_experts, int *cold, int *flags, cudaStream_t s) {
    cold_routes_kernel<<<1, 1, 0, s>>>(ids, k, bound, n_experts, cold, flags);
    note_launch();
    return cudaGetLastError();
}

__global__ void add_rows_kernel(const int64_t *a, const int64_t *b, int64_t *out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (int64_t)((uint64_t)a[i] + (uint64_t)b[i]);
}

cudaError_t launch_add_rows(const int64_t *a, const int64_t *b, int64_t *out, long long n, cudaStream_t s) {
    add_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, b, out, n);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_limbs(const int64_t *x, long long n_rows, long long K, int8_t *planes, int *flags, cudaStream_t s,
                         int *nl_out, int *clear0, int *clear1, int64_t *zero, long long zero_n, int8_t *sums) {
    const LimbClears clears = {clear0, clear1, zero, zero ? zero_n : 0, sums, (int)((K / 32 + 31) / 32 * 32)};
    if (sums && (K % 256 || (reinterpret_cast<uintptr_t>(x) & 15))) return cudaErrorInvalidValue;
    if (K % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(planes) & 7) == 0)
        launch_behind(sums ? limbs8_kernel<true> : limbs8_kernel<false>, grid_for(n_rows * (K >> 3), 256), 256, 0, s, x, n_rows, K, planes, flags, nl_out, clears);
    else
        launch_behind(limbs_kernel, grid_for(n_rows * K, 256), 256, 0, s, x, n_rows, K, planes, flags, nl_out, clears);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_exact_linear(const uint8_t *w, int qtype, long long out_f, long long nb, const int64_t *x,
                                long long T, int fw, int64_t *out, cudaStream_t s) {
    const long long n = out_f * T;
    exact_linear_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(w, qtype, out_f, nb, x, T, fw, out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_exact_dense(const int64_t *w, long long out_f, long long in_f, const int64_t *x, long long T,
                               int fw, int64_t *out, int *flags, cudaStream_t s) {
    const long long n = out_f * T * 32;
    exact_dense_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(w, out_f, in_f, x, T, fw, out, flags);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_silu_mul(int64_t *a, const int64_t *b, long long n, int fa, cudaStream_t s) {
    silu_mul_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, b, n, fa);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_combine(const int64_t *dn, const int64_t *gates, long long T, int k, long long d_model, int fa,
                           int64_t *out, cudaStream_t s) {
    const long long n = T * d_model;
    combine_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dn, gates, T, k, d_model, fa, out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_topk(const int64_t *logits, long long rows, int n_experts, int k, int fa, int *ids, int64_t *gates,
                        cudaStream_t s) {
    if (n_experts > 1024 || n_experts <= 0 || k <= 0) return cudaErrorInvalidValue;
    const long long n = rows * 32;
    launch_behind(topk_kernel, (unsigned)((n + 127) / 128), 128, 0, s, logits, rows, n_experts, k, fa, ids, gates);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_rmsnorm(const int64_t *x, long long rows, long long width, const int64_t *gain, int fa,
                           unsigned long long eps, int64_t *out, int *flags, cudaStream_t s) {
    if (rows <= 0 || width <= 0 || width > (1 << 30)) return cudaErrorInvalidValue;
    return launch_norm({x, rows, rows, (int)width, 0, false, gain, nullptr, fa, eps, out, nullptr, flags, PlaneDuties()}, s);
}

cudaError_t launch_rmsnorm_pair(const int64_t *x, long long rows_a, long long rows_b, long long width, const int64_t *gain_a,
                                const int64_t *gain_b, int fa, unsigned long long eps, int64_t *out, int *flags, cudaStream_t s) {
    if (rows_a + rows_b <= 0 || width <= 0 || width > (1 << 30)) return cudaErrorInvalidValue;
    return launch_norm({x, rows_a + rows_b, rows_a, (int)width, 0, false, gain_a, gain_b, fa, eps, out, nullptr, flags, PlaneDuties()}, s);
}

cudaError_t launch_rmsnorm_planes(const int64_t *x, long long rows, long long width, const int64_t *gain, int fa,
                                  unsigned long long eps, int64_t *out, int8_t *planes, int *flags, const PlaneDuties &duties, cudaStream_t s) {
    if (rows <= 0 || width <= 0 || (width & 127) || width > (1 << 30) || !planes) return cudaErrorInvalidValue;
    return launch_norm({x, rows, rows, (int)width, 0, false, gain, nullptr, fa, eps, out, planes, flags, duties}, s);
}

cudaError_t launch_dispatch(const int *ids, const int64_t *gates, long long T, int k, int n_experts, int *grp_off,
                            int *pair_tok, int64_t *pair_gate, cudaStream_t s, int expert_base) {
    if (n_experts > 1024 || n_experts <= 0) return cudaErrorInvalidValue;
    const int warps = n_experts <= 320 ? 32 : 8;                        // cnt[warps][E] + start[E + 1] stays below 48 KB
    const size_t smem = ((size_t)warps * n_experts + n_experts + 1) * sizeof(int);
    launch_behind(dispatch_kernel, 1, 32 * warps, smem, s, ids, gates, T, k, n_experts, expert_base, grp_off, pair_tok, pair_gate);
    note_launch();
    return cudaGetLastError();
}

}  // namespace iie
