// Q1_0 (one sign bit per weight, one integer scale per 128-weight block) linear products.
//
// Contract (bonsai/src/trinote/infer_int/reference_bonsai.py:149-219, bonsai/tools/bonsai_q1_kernel.c:85-106,
// bonsai/tools/bonsai_q1_gpu.cu:78-123):
//     out[t,o] = sum_b arshift( (sum_{i<128} s_i x[t,128b+i]) * scale[o,b]  mod 2^64, frac )        (mod 2^64)
// with s_i = +1 for a set bit (little-endian inside each byte) and -1 for a clear one, the shift flooring
// toward minus infinity and applied per block BEFORE the blocks are added.
//
// The reference spends one warp on every (token, row) output and adds 128 int64 values per block on the
// CUDA cores.  Here the block sums run on the tensor cores and stay exact modulo 2^64:
//   * sum_i s_i x_i = 2 * P - S with P = sum over set bits of x_i and S = sum_i x_i; S does not depend on
//     the weight row and is formed once per (token, block) while the activations are split into digits;
//   * x = sum_l 256^l d_l (mod 2^64) with eight balanced digits d_l in [-128,127] (the carry out of the
//     eighth digit is a multiple of 2^64 and drops out), so P = sum_l 256^l sum_i bit_i d_{l,i} (mod 2^64):
//     the eight digit planes are the N = 8 columns of an int8 warp MMA whose A operand is the weight
//     bits expanded to bytes 0/1.  |sum_i bit_i d_{l,i}| <= 128*128, far inside int32.  Every int64 input
//     is therefore handled exactly; there is no envelope and no fallback.
//
// Weight layout ("units"): rows are grouped in tiles of 16; unit (tile, block) holds 256 bytes of sign
// bits in MMA A-fragment order followed by the 16 block scales (int32 when every scale of the matrix
// fits, else int64).  Lane (g,t) owns two 32-bit words; bit r + 8 i of word mp is the sign bit of row
// g + 8 (r & 1), column 32 (2 mp + (r >> 2)) + 8 t + 4 ((r >> 1) & 1) + i, so A register j of MMA m is
// (word[m >> 1] >> (4 (m & 1) + j)) & 0x01010101: two instructions per register.
#include "kernels.h"
#include "mma_items.cuh"

namespace iie {

namespace {

__device__ __forceinline__ int64_t q1_shift(int64_t v, int sh) { return v >> sh; }   // arithmetic: floors

// ---- registration: raw [out_f][nb][16] bits + [out_f][nb] scales -> units ------------------------------------
template <typename ST, typename DT>
__global__ void q1_repack_kernel(const uint8_t *bits, const ST *scale, long long out_f, long long nb, long long n_tiles,
                                 uint8_t *units, unsigned long long *max_scale) {
    constexpr int US = 256 + 16 * (int)sizeof(DT);
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;     // (tile, block, slot 0..79)
    const long long n = n_tiles * nb * 80;
    if (idx >= n) return;
    const int slot = (int)(idx % 80);
    const long long tb = idx / 80, tile = tb / nb, b = tb - tile * nb;
    uint8_t *unit = units + tb * US;
    if (slot < 64) {
        const int lane = slot >> 1, mp = slot & 1, g = lane >> 2, t = lane & 3;
        uint32_t w = 0;
        for (int p = 0; p < 32; p++) {
            const int r = p & 7, i = p >> 3;
            const long long row = tile * 16 + g + 8 * (r & 1);
            const int k = 32 * (2 * mp + (r >> 2)) + 8 * t + 4 * ((r >> 1) & 1) + i;
            if (row < out_f) w |= (uint32_t)((bits[(row * nb + b) * 16 + (k >> 3)] >> (k & 7)) & 1) << p;
        }
        reinterpret_cast<uint32_t *>(unit)[lane * 2 + mp] = w;
    } else {
        const int r = slot - 64;
        const long long row = tile * 16 + r;
        const long long sc = row < out_f ? (long long)scale[row * nb + b] : 0;
        const unsigned long long mag = sc < 0 ? 0ULL - (unsigned long long)sc : (unsigned long long)sc;
        reinterpret_cast<DT *>(unit + 256)[r] = (DT)sc;
        if (mag > *(volatile unsigned long long *)max_scale) atomicMax(max_scale, mag);
    }
}

// ---- activations: digit planes [tok][8][K], digits in use ---------------------------
// With `up` the activation is the SwiGLU of two rows of width K: ((x * sigmoid(x)) >> frac) * up >> frac, wrapping products;
// x and up then advance by `ld` per token.  `wide`: every row starts on 16 bytes.
__device__ __forceinline__ void q1_four(const int64_t *src, bool wide, int64_t (&v)[4]) {
    longlong2 a, b;
    if (wide) { a = *reinterpret_cast<const longlong2 *>(src); b = *reinterpret_cast<const longlong2 *>(src + 2); }
    else { a = make_longlong2(src[0], src[1]); b = make_longlong2(src[2], src[3]); }
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__global__ void q1_prep_kernel(const int64_t *x, const int64_t *up, long long ld, bool wide, int frac, int64_t log2e, int64_t clip, long long T,
                               long long nb, int8_t *planes, const PlaneDuties duties) {
    pdl_enter();
    int *nl_out = duties.nl;
    if (duties.nl_clear && blockIdx.x == 0 && threadIdx.x == 0) *duties.nl_clear = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < duties.zero_n; i += (long long)gridDim.x * blockDim.x) duties.zero[i] = 0;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= T * nb) return;
    const long long tok = wid / nb, b = wid - tok * nb, K = nb * 128;
    const int64_t *src = x + tok * (up ? ld : K) + b * 128 + lane * 4;
    int64_t v[4];
    q1_four(src, wide, v);
    if (up) {
        const int64_t *us = up + tok * ld + b * 128 + lane * 4;
        int64_t u[4];
        q1_four(us, wide, u);
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = silu_up_wrapped(v[i], u[i], frac, log2e, clip);
    }
    uint32_t pl[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    int nl = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        bool ok;
        const uint64_t d = balanced_digits8(v[i], ok);
        nl = max(nl, ok ? digits_used(d) : 9);
#pragma unroll
        for (int l = 0; l < 8; l++) pl[l] |= (uint32_t)((d >> (8 * l)) & 0xFF) << (8 * i);
    }
#pragma unroll
    for (int l = 0; l < 8; l++) *reinterpret_cast<uint32_t *>(planes + (tok * 8 + l) * K + b * 128 + lane * 4) = pl[l];
    nl = __reduce_max_sync(0xffffffffu, nl);
    if (lane == 0 && nl_out && nl > *(volatile int *)nl_out) atomicMax(nl_out, nl);
}

// SiLU(gate) * up with the wrapping products of bonsai/src/trinote/infer_int/reference_bonsai.py:246-262,611-614:
// silu = (gate * sigmoid(gate)) >> frac and h = (silu * up) >> frac, both products modulo 2^64.
__global__ void q1_silu_mul_kernel(const int64_t *gate, const int64_t *up, long long n, int frac, int64_t log2e, int64_t clip,
                                   int64_t *out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = silu_up_wrapped(gate[i], up[i], frac, log2e, clip);
}

// one row of a registered Q1_0 matrix as int64: sign * block scale (reference_bonsai.py:138-146 q1_rows_fp)
template <typename DT>
__global__ void q1_embed_row_kernel(const uint8_t *units, long long nb, const int *row_dev, long long row_host, int64_t *out) {
    constexpr int US = 256 + 16 * (int)sizeof(DT);
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nb * 128) return;
    const long long row = row_dev ? (long long)*row_dev : row_host, b = k >> 7;
    const int kk = (int)(k & 127), rloc = (int)(row & 15), g = rloc & 7, hi = rloc >> 3;
    const int m = kk >> 5, t = (kk & 31) >> 3, jj = ((kk & 31) >> 2) & 1, i = kk & 3;
    const int r = (m & 1) * 4 + ((jj << 1) | hi), mp = m >> 1;
    const uint8_t *unit = units + ((row >> 4) * nb + b) * US;
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(unit) + (4 * g + t) * 2 + mp);
    const int64_t sc = (int64_t)__ldg(reinterpret_cast<const DT *>(unit + 256) + rloc);
    out[k] = ((w >> (r + 8 * i)) & 1u) ? sc : -sc;
}

}  // namespace

size_t q1_unit_bytes(bool sc32) { return 256 + 16 * (sc32 ? 4 : 8); }

cudaError_t launch_q1_repack(const uint8_t *bits, const void *scale, int src_bits, bool sc32, long long out_f, long long nb,
                             uint8_t *units, unsigned long long *max_scale, cudaStream_t s) {
    const long long n_tiles = (out_f + 15) / 16, n = n_tiles * nb * 80;
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (src_bits == 64 && !sc32) q1_repack_kernel<long long, long long><<<grid, 256, 0, s>>>(bits, (const long long *)scale, out_f, nb, n_tiles, units, max_scale);
    else if (src_bits == 64) q1_repack_kernel<long long, int><<<grid, 256, 0, s>>>(bits, (const long long *)scale, out_f, nb, n_tiles, units, max_scale);
    else if (sc32) q1_repack_kernel<int, int><<<grid, 256, 0, s>>>(bits, (const int *)scale, out_f, nb, n_tiles, units, max_scale);
    else return cudaErrorInvalidValue;
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_q1_prep(const int64_t *x, long long T, long long nb, int8_t *planes, const PlaneDuties &duties,
                           cudaStream_t s) {
    const long long warps = T * nb;
    launch_behind(q1_prep_kernel, (unsigned)((warps * 32 + 255) / 256), 256, 0, s, x, nullptr, 0, (reinterpret_cast<uintptr_t>(x) & 15) == 0, 0, 0, 0, T, nb, planes, duties);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_q1_prep_swiglu(const int64_t *gate, const int64_t *up, long long ld, int frac, long long T, long long nb,
                                  int8_t *planes, const PlaneDuties &duties, cudaStream_t s) {
    if (!gate || !up || frac < 1 || frac > 29) return cudaErrorInvalidValue;
    const long long warps = T * nb;
    const bool wide = ((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | (uintptr_t)(ld * 8)) & 15) == 0;
    launch_behind(q1_prep_kernel, (unsigned)((warps * 32 + 255) / 256), 256, 0, s, gate, up, ld, wide, frac, sigmoid_log2e(frac), sigmoid_clip(frac), T, nb,
                                                                        planes, duties);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_q1_apply(const Q1Part *parts, int n_parts, bool sc32, long long nb, const int8_t *planes, long long T, long long frac,
                            const int *nl, cudaStream_t s) {
    if (n_parts < 1 || nb <= 0 || T <= 0) return cudaErrorInvalidValue;
    return launch_q1_tc(parts, n_parts, sc32, nb, planes, T, frac <= 0 ? 0 : (frac >= 63 ? 63 : (int)frac), nl, s);
}

cudaError_t launch_q1_silu_mul(const int64_t *gate, const int64_t *up, long long n, int frac, int64_t *out, cudaStream_t s) {
    if (n <= 0 || frac < 1 || frac > 29) return cudaErrorInvalidValue;
    q1_silu_mul_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(gate, up, n, frac, sigmoid_log2e(frac), sigmoid_clip(frac), out);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_q1_embed_row(const uint8_t *units, bool sc32, long long nb, const int *row_dev, long long row_host, int64_t *out,
                                cudaStream_t s) {
    const unsigned grid = (unsigned)((nb * 128 + 255) / 256);
    if (sc32) q1_embed_row_kernel<int><<<grid, 256, 0, s>>>(units, nb, row_dev, row_host, out);
    else q1_embed_row_kernel<long long><<<grid, 256, 0, s>>>(units, nb, row_dev, row_host, out);
    note_launch();
    return cudaGetLastError();
}

}  // namespace iie
