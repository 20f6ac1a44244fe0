// Exact integer attention of the new tokens of independent sequences over their caches (arithmetic: attn.cu), one thread-block
// cluster per (sequence, KV head).
//
// The softmax needs the maximum and the normaliser of all visible keys before the values count, so the keys are cut among the CTAs
// of a cluster, scores and exponentials stay in shared memory, and maximum, normaliser and output sums pass through distributed
// shared memory: keys and values are read once, nothing else goes to memory, and a cluster barrier takes the place of a grid barrier.
//
// A warp works on its own 32-key tiles without barriers; keys and values go from memory straight into the fragments of the eight-bit
// tensor cores (every int32 is its four bytes, every product exact), the next step's loads under way while one is multiplied.
// Scores: 16 keys x 8 heads x 32 dimensions per step.  Values: probabilities are bytes too; the low bytes of the eight heads are rows
// 0..7 of the operand, the second bytes rows 8..15, and columns are taken so that one 16-byte load of a value row feeds four steps.
//
// What bounds it: 64 sequences of 4096 keys, 4 KV heads of 128 (1.07 GB): 258 us; the copies alone take 164, the rest is the latency of
// eight warps per SM (their registers hold the loads under way: with twelve warps and less of it 330), about 1800 instructions per
// tile.  Three kernels with the scores in memory took 540.  A call for one sequence goes to attn_fat_kernel, whose chain is shorter than
// one warp's over a tile (12 against 16 us at 513 keys); a batched call comes here whatever its number of sequences.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "mma_items.cuh"
#include "norm.cuh"
#include "softmax.cuh"

namespace cg = cooperative_groups;

namespace iie {

namespace {

constexpr int AC_WARPS = 4, AC_THREADS = 32 * AC_WARPS;
constexpr int AC_TILE = 32;                    // keys of a tile
constexpr int AC_HEADS = 8;                    // query heads of a KV head at most
constexpr int AC_MAX_CLUSTER = 8;
constexpr int AC_AHEAD = 1;                    // tiles of a warp that are on their way to the cache ahead of the one at hand
constexpr int AC_MAX_TILES = 64;               // tiles of a CTA: two CTAs then fit an SM

template <int HD>
__host__ __device__ constexpr size_t ac_smem(int tiles) {          // scores [8][32 tiles + 4] and queries as int64, later the warps' sums [4][8][HD]; queries as bytes; the new key
    const size_t a = (size_t)AC_HEADS * (tiles * AC_TILE + 4) * 4 + (size_t)AC_HEADS * HD * 8, b = (size_t)AC_WARPS * AC_HEADS * HD * 8;
    return (a > b ? a : b) + (size_t)4 * AC_HEADS * (HD + 16) + (size_t)HD * 8;
}

// rows that a later tile reads, on their way from memory to the cache: one request per tile
__device__ __forceinline__ void ac_ahead(const int32_t *rows, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(rows), "r"(bytes) : "memory");
}
__device__ __forceinline__ int4 ac_load(const int32_t *p) { return __ldcg(reinterpret_cast<const int4 *>(p)); }

// the four bytes of four consecutive values, transposed: d[b] = byte b of (x, y, z, w)
__device__ __forceinline__ void ac_bytes(uint32_t x, uint32_t y, uint32_t z, uint32_t w, uint32_t (&d)[4]) {
    const uint32_t t0 = __byte_perm(x, y, 0x5140), t1 = __byte_perm(x, y, 0x7362), t2 = __byte_perm(z, w, 0x5140), t3 = __byte_perm(z, w, 0x7362);
    d[0] = __byte_perm(t0, t2, 0x5410); d[1] = __byte_perm(t0, t2, 0x7632); d[2] = __byte_perm(t1, t3, 0x5410); d[3] = __byte_perm(t1, t3, 0x7632);
}
// D(16x8,s32) = A(16x32, 8-bit, row) * B(32x8, 8-bit, col) (+ D), the operands signed or not.  (An unsigned B costs two instructions.)
template <bool AS>
__device__ __forceinline__ void ac_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (AS)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool BS>
__device__ __forceinline__ void ac_mma_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (BS)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

__device__ __forceinline__ void ac_rotate(const AttnArgs &a, long long pos, int i, int64_t &x0, int64_t &x1) {
    if (!a.rope) return;
    const int half = a.hd / 2;
    const int64_t c = a.cos[pos * half + i], s = a.sin[pos * half + i];
    const int64_t y0 = (x0 * c - x1 * s) >> a.fa, y1 = (x0 * s + x1 * c) >> a.fa;
    x0 = y0; x1 = y1;
}

template <int HD, bool SHORT>                                      // SHORT: fa <= 16, exponentials and probabilities of 32-bit products
__global__ void __launch_bounds__(AC_THREADS, 2) attn_cluster_kernel(const AttnArgs a) {
    using Exp = std::conditional_t<SHORT, SoftmaxExp16, SoftmaxExp>;
    using Quotient = std::conditional_t<SHORT, SoftmaxQuotient16, SoftmaxQuotient>;
    pdl_enter();
    constexpr int QLD = HD + 16, HALF = HD / 2;
    extern __shared__ __align__(128) unsigned char ac_sm[];
    __shared__ long long s_max[AC_WARPS][AC_HEADS], s_base[AC_WARPS][AC_HEADS];
    __shared__ unsigned long long s_z[AC_WARPS][AC_HEADS];
    __shared__ int s_wide;
    cg::cluster_group cluster = cg::this_cluster();
    const int n_c = (int)gridDim.x, rank = (int)blockIdx.x, kv = blockIdx.y, seq = blockIdx.z, rep = a.H / a.Hkv;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const long long pos = a.pos_each ? (long long)a.pos_each[seq] : a.pos;
    if (a.pos_each && (pos < 0 || pos > a.pos || pos >= a.Lmax)) {          // the whole cluster
        if (tid == 0 && rank == 0 && kv == 0) atomicOr(a.flags, 16);
        return;
    }
    const long long lo = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int n_keys = (int)(pos - lo + 1), n_tiles = (n_keys + AC_TILE - 1) / AC_TILE, per = (n_tiles + n_c - 1) / n_c;      // per <= a.chunk
    const int first = min(rank * per, n_tiles), end = min(first + per, n_tiles), stride = a.chunk * AC_TILE + 4;
    const bool own = first < end && end == n_tiles;                         // this CTA appends the new row
    int32_t *off = reinterpret_cast<int32_t *>(ac_sm);                      // [8][stride]: scores, then exponentials
    int64_t *q64 = reinterpret_cast<int64_t *>(off + AC_HEADS * stride);   // rotated queries [8][HD] (rows beyond rep are zero)
    int8_t *qd = reinterpret_cast<int8_t *>(ac_sm + ac_smem<HD>(a.chunk) - HD * 8 - 4 * AC_HEADS * QLD);      // their balanced digits [4][8][HD + 16]
    int64_t *knew = reinterpret_cast<int64_t *>(qd + 4 * AC_HEADS * QLD);   // the new key, normed
    const int32_t *kc = a.kcache + (long long)seq * a.seq_stride + ((long long)kv * a.Lmax + lo) * HD;
    const int32_t *vc = a.vcache + (long long)seq * a.seq_stride + ((long long)kv * a.Lmax + lo) * HD;
    // tile `tile` of the keys, or of the values behind the warp's last key tile; rows that the cache held before this token
    const int mine = first + warp < end ? (end - first - warp + AC_WARPS - 1) / AC_WARPS : 0;      // tiles of this warp
    auto ahead = [&](int i) {
        const int32_t *cache = i < mine ? kc : vc;
        const int tile = first + warp + AC_WARPS * (i < mine ? i : i - mine), rows = min(AC_TILE, n_keys - 1 - tile * AC_TILE);
        if (lane == 0 && i < 2 * mine && rows > 0) ac_ahead(cache + (long long)tile * AC_TILE * HD, (uint32_t)(rows * HD * 4));
    };
#pragma unroll
    for (int i = 0; i < AC_AHEAD; i++) ahead(i);
    if (tid == 0) s_wide = 0;
    if (lane < AC_HEADS) s_base[warp][lane] = 0;                            // (no tile: never used)
    // ---- per-head norms where the caller wants them here, rotation, bytes of the queries; the new row into the cache ----------------
    const long long kv_row = (long long)seq * (a.kv_ld ? a.kv_ld : (long long)a.Hkv * HD) + (long long)kv * HD;
    const int64_t *q_in = a.q + (long long)seq * (a.q_ld ? a.q_ld : (long long)a.H * HD) + (long long)kv * rep * HD, *k_in = a.k + kv_row, *v_in = a.v + kv_row;
    if (a.qgain) {
        for (int r = warp; r < rep + (own ? 1 : 0); r += AC_WARPS) {
            const int64_t *src = r == rep ? k_in : q_in + r * HD, *gain = r == rep ? a.kgain : a.qgain;
            int64_t *dst = r == rep ? knew : q64 + r * HD;
            int64_t x[HD / 32], gv[HD / 32];
            u128 ssq = 0;
            uint64_t mx = 0, gm = 0;
#pragma unroll
            for (int k = 0; k < HD / 32; k++) { x[k] = src[lane + 32 * k]; gv[k] = gain[lane + 32 * k]; }
#pragma unroll
            for (int k = 0; k < HD / 32; k++) {
                const uint64_t m = uabs64(x[k]), ga = uabs64(gv[k]);
                if ((m >> 32) == 0) ssq += (uint64_t)(uint32_t)m * (uint32_t)m; else ssq += (u128)m * m;
                mx = m > mx ? m : mx; gm = ga > gm ? ga : gm;
            }
            const uint32_t xb = __reduce_max_sync(0xffffffffu, (uint32_t)(64 - __clzll((long long)mx)) | (mx > (1ULL << 57) ? 128u : 0u));
            const uint32_t gb = __reduce_max_sync(0xffffffffu, (uint32_t)(64 - __clzll((long long)gm)));
            const NormRow n(warp_sum128(ssq), (int)(xb & 127u), (int)gb, (xb & 128u) != 0, HD, a.eps, a.fa, true);
            bool bad = n.refused;
            if (n.fast || n.refused) {
#pragma unroll
                for (int k = 0; k < HD / 32; k++) dst[lane + 32 * k] = n.refused ? 0 : n.fast_value((int)x[k], (int)gv[k]);
            } else {
                const uint64_t inv = n.rms < (1ULL << 62) ? recip_below(n.rms) : 0, gmax = warp_gain_max(gain, HD);
#pragma unroll 1
                for (int i = lane; i < HD; i += 32) dst[i] = norm_value(src[i], n.rms, inv, gmax, gain[i], true, a.fa, bad);
            }
            if (bad) atomicOr(a.flags, 2);
        }
    }
    __syncthreads();                                                        // norms and the words set above
    bool wide = false;                                                      // a query beyond four balanced digits
    for (int idx = tid; idx < AC_HEADS * HALF; idx += AC_THREADS) {
        const int r = idx / HALF, i = idx - r * HALF;
        const int i0 = a.rope == 2 ? i : 2 * i, i1 = a.rope == 2 ? i + HALF : 2 * i + 1;
        int64_t x0 = 0, x1 = 0;
        if (r < rep) {
            const int64_t *src = a.qgain ? q64 + r * HD : q_in + r * HD;    // in place: a pair is one thread's
            x0 = src[i0]; x1 = src[i1];
            ac_rotate(a, pos, i, x0, x1);
        }
        q64[r * HD + i0] = x0; q64[r * HD + i1] = x1;
        const uint32_t d0 = ((uint32_t)x0 + 0x80808080u) ^ 0x80808080u, d1 = ((uint32_t)x1 + 0x80808080u) ^ 0x80808080u;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            qd[(b * AC_HEADS + r) * QLD + i0] = (int8_t)(d0 >> (8 * b));
            qd[(b * AC_HEADS + r) * QLD + i1] = (int8_t)(d1 >> (8 * b));
        }
        wide |= x0 < -0x80808080LL || x0 > 0x7F7F7F7FLL || x1 < -0x80808080LL || x1 > 0x7F7F7F7FLL;
    }
    if (wide) s_wide = 1;
    if (own) {                                                              // a 128-thread CTA: one value and at most one pair each
        bool bad = false;
        int32_t *kd = a.kcache + (long long)seq * a.seq_stride + ((long long)kv * a.Lmax + pos) * HD;
        int32_t *vd = a.vcache + (long long)seq * a.seq_stride + ((long long)kv * a.Lmax + pos) * HD;
        if (tid < HALF) {
            const int i0 = a.rope == 2 ? tid : 2 * tid, i1 = a.rope == 2 ? tid + HALF : 2 * tid + 1;
            const int64_t *src = a.qgain ? knew : k_in;
            int64_t x0 = src[i0], x1 = src[i1];
            ac_rotate(a, pos, tid, x0, x1);
            bad = x0 != (int32_t)x0 || x1 != (int32_t)x1;
            kd[i0] = (int32_t)x0; kd[i1] = (int32_t)x1;
        }
        if (tid < HD) { const int64_t x = v_in[tid]; bad = bad || x != (int32_t)x; vd[tid] = (int32_t)x; }
        if (bad) atomicOr(a.flags, 4);
    }
    __syncthreads();
    const bool use_wide = s_wide != 0;

    // ---- pass 1: scores of this warp's tiles, as 32-bit distances from a base per head: the first tile's maximum; a score more than 2^31
    //      above moves it and the distances so far, one more than 2^31 below is beyond every exponential's reach and stays at the edge ---
    const int last = n_keys - 1;                                            // rows past it are read as it
    long long best[2] = {INT64_MIN, INT64_MIN};                            // heads 2t, 2t + 1
    // this warp's scores of head h so far, which its lanes stored in another order, move to another base
    auto rebase = [&](int h, long long to, int tiles_done) {
        __syncwarp();
        const long long by = to - s_base[warp][h];
        for (int j = 0; j <= tiles_done; j++) {
            int32_t *e = off + h * stride + (warp + AC_WARPS * j) * AC_TILE + lane;
            *e = (int32_t)max((long long)*e - by, (long long)INT32_MIN);
        }
        __syncwarp();
        if (lane == 0) s_base[warp][h] = to;
        __syncwarp();
    };
    auto put = [&](int h, int local, long long score) {                    // local: key of the CTA
        off[h * stride + local] = (int32_t)max(score - s_base[warp][h], (long long)INT32_MIN);      // (rows past the last hold anything)
    };
    int j = 0;
    // key rows g and g + 8 of group i of sixteen (two per tile), dimensions 4t .. and 16 + 4t .. of every 32
    auto key_rows = [&](int i, const int32_t *&ra, const int32_t *&rb) {
        const int key = (first + warp + AC_WARPS * (i >> 1)) * AC_TILE + 16 * (i & 1) + g;
        ra = kc + (long long)min(key, last) * HD + 4 * t; rb = kc + (long long)min(key + 8, last) * HD + 4 * t;
    };
    int4 k[HD / 32][4];                                                     // the group at hand; every step's place takes the next group's load
    if (!use_wide && mine > 0) {
        const int32_t *ra, *rb;
        key_rows(0, ra, rb);
#pragma unroll
        for (int st = 0; st < HD / 32; st++) {
            k[st][0] = ac_load(ra + 32 * st); k[st][1] = ac_load(rb + 32 * st); k[st][2] = ac_load(ra + 32 * st + 16); k[st][3] = ac_load(rb + 32 * st + 16);
        }
    }
    for (int tile = first + warp; tile < end; tile += AC_WARPS, j++) {
        ahead(j + AC_AHEAD);
        const int left = n_keys - tile * AC_TILE, local0 = (tile - first) * AC_TILE;      // visible keys of the tile
        if (!use_wide) {
            long long sc[2][4];
#pragma unroll 1
            for (int mt = 0; mt < 2; mt++) {
                int acc[7][4];
#pragma unroll
                for (int i = 0; i < 7; i++) { acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0; }
                const int32_t *ra, *rb;
                key_rows(min(2 * j + mt + 1, 2 * mine - 1), ra, rb);
#pragma unroll
                for (int st = 0; st < HD / 32; st++) {
                    const int4 k0 = k[st][0], k1 = k[st][1], k2 = k[st][2], k3 = k[st][3];
                    k[st][0] = ac_load(ra + 32 * st); k[st][1] = ac_load(rb + 32 * st); k[st][2] = ac_load(ra + 32 * st + 16); k[st][3] = ac_load(rb + 32 * st + 16);
                    uint32_t A0[4], A1[4], A2[4], A3[4];
                    ac_bytes(k0.x, k0.y, k0.z, k0.w, A0); ac_bytes(k1.x, k1.y, k1.z, k1.w, A1);
                    ac_bytes(k2.x, k2.y, k2.z, k2.w, A2); ac_bytes(k3.x, k3.y, k3.z, k3.w, A3);
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        const int8_t *qb = qd + (b * AC_HEADS + g) * QLD + 32 * st + 4 * t;
                        const uint32_t b0 = *reinterpret_cast<const uint32_t *>(qb), b1 = *reinterpret_cast<const uint32_t *>(qb + 16);
                        ac_mma<false>(acc[b], A0[0], A1[0], A2[0], A3[0], b0, b1);
                        ac_mma<false>(acc[b + 1], A0[1], A1[1], A2[1], A3[1], b0, b1);
                        ac_mma<false>(acc[b + 2], A0[2], A1[2], A2[2], A3[2], b0, b1);
                        ac_mma<true>(acc[b + 3], A0[3], A1[3], A2[3], A3[3], b0, b1);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    long long dot = 0;
#pragma unroll
                    for (int w = 6; w >= 0; w--) dot = dot * 256 + (long long)acc[w][i];
                    const long long s = ((dot >> a.fa) * a.inv_sqrt) >> a.fa;
                    if (mt) sc[1][i] = s; else sc[0][i] = s;
                }
            }
            bool far = false;
            long long top[2] = {INT64_MIN, INT64_MIN};
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (16 * (i >> 2) + g + ((i & 2) ? 8 : 0) < left) top[i & 1] = max(top[i & 1], sc[i >> 2][i & 3]);
            if (j == 0) {                                                   // the first tile's maximum is the first base
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    long long m = top[i];
#pragma unroll
                    for (int s2 = 4; s2 < 32; s2 <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s2));
                    if (g == 0) s_base[warp][2 * t + i] = m;
                }
                __syncwarp();
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                best[i] = max(best[i], top[i]);
                far = far || (top[i] != INT64_MIN && top[i] - s_base[warp][2 * t + i] > INT32_MAX);
            }
            if (__any_sync(0xffffffffu, far)) {
#pragma unroll 1
                for (int h = 0; h < AC_HEADS; h++) {
                    long long m = (h >> 1) == t ? ((h & 1) ? top[1] : top[0]) : INT64_MIN;
#pragma unroll
                    for (int s2 = 16; s2 > 0; s2 >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s2));
                    if (m != INT64_MIN && m - s_base[warp][h] > INT32_MAX) rebase(h, m, j - 1);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++) put(2 * t + (i & 1), local0 + 16 * (i >> 2) + g + ((i & 2) ? 8 : 0), sc[i >> 2][i & 3]);
        } else {
            // a query value beyond int32: wrapping 64-bit products, a key per lane (four values a load, four loads under way: 38 sequences of
            // 602 keys, 12 heads over 2: 92 us; value by value 318, the three kernels with the scores in memory 148)
            const int32_t *kr = kc + (long long)min(tile * AC_TILE + lane, last) * HD;
#pragma unroll 1
            for (int h = 0; h < AC_HEADS; h++) {
                long long dot = 0;
                if (h < rep && lane < left) {
                    const longlong2 *qr = reinterpret_cast<const longlong2 *>(q64 + h * HD);
#pragma unroll 4
                    for (int i = 0; i < HD / 4; i++) {
                        const int4 kv = ac_load(kr + 4 * i);
                        const longlong2 qa = qr[2 * i], qb = qr[2 * i + 1];
                        dot += qa.x * (long long)kv.x + qa.y * (long long)kv.y + qb.x * (long long)kv.z + qb.y * (long long)kv.w;
                    }
                }
                const long long s = ((dot >> a.fa) * a.inv_sqrt) >> a.fa;
                long long m = lane < left ? s : INT64_MIN;
#pragma unroll
                for (int s2 = 16; s2 > 0; s2 >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, s2));
                if ((h >> 1) == t) { if (h & 1) best[1] = max(best[1], m); else best[0] = max(best[0], m); }
                if (j == 0 || m - s_base[warp][h] > INT32_MAX) rebase(h, m, j - 1);
                put(h, local0 + lane, s);
            }
        }
    }
    // ---- the row maximum over the cluster: lane l takes head l % 8 of warp l / 8 of every CTA ------------------------------------
#pragma unroll
    for (int i = 0; i < 2; i++) {
#pragma unroll
        for (int s2 = 4; s2 < 32; s2 <<= 1) best[i] = max(best[i], __shfl_xor_sync(0xffffffffu, best[i], s2));
        if (g == 0) s_max[warp][2 * t + i] = best[i];
    }
    cluster.sync();
    const int head8 = lane & 7, from = lane >> 3;
    long long m_all = INT64_MIN;
    for (int r = 0; r < n_c; r++) m_all = max(m_all, cluster.map_shared_rank(&s_max[from][head8], r)[0]);
    m_all = max(m_all, __shfl_xor_sync(0xffffffffu, m_all, 8));
    m_all = max(m_all, __shfl_xor_sync(0xffffffffu, m_all, 16));
    const long long above = __shfl_sync(0xffffffffu, m_all, g) - s_base[warp][g];      // from here on a lane has head g, keys 8t .. 8t + 7 of a tile
    // ---- pass 2: exponentials over the scores, their sum --------------------------------------------------------------------------
    const Exp exp2(a.fa, a.log2e, a.clip);
    unsigned long long z = 0;
    for (int tile = first + warp; tile < end; tile += AC_WARPS) {
        int4 *e4 = reinterpret_cast<int4 *>(off + g * stride + (tile - first) * AC_TILE + 8 * t);
        const int left = n_keys - tile * AC_TILE - 8 * t;
        const int4 lo4 = e4[0], hi4 = e4[1];
        int e[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int v = SHORT ? (int)exp2((uint32_t)min(above - e[i], a.clip)) : (int)exp2(above - e[i]);
            e[i] = i < left && g < rep ? v : 0;
            z += (unsigned)e[i];
        }
        e4[0] = make_int4(e[0], e[1], e[2], e[3]); e4[1] = make_int4(e[4], e[5], e[6], e[7]);
    }
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    if (t == 0) s_z[warp][g] = z;
    cluster.sync();
    unsigned long long z_all = 0;
    for (int r = 0; r < n_c; r++) z_all += cluster.map_shared_rank(&s_z[from][head8], r)[0];
    z_all += __shfl_xor_sync(0xffffffffu, z_all, 8);
    z_all += __shfl_xor_sync(0xffffffffu, z_all, 16);
    z = __shfl_sync(0xffffffffu, z_all, g);
    const Quotient quotient(g < rep ? z : 0, a.fa);
    // ---- pass 3: probabilities floor(e 2^fa / z) as bytes, times the values --------------------------------------------------------
    long long sum[HD / 8][2];
#pragma unroll
    for (int i = 0; i < HD / 8; i++) sum[i][0] = sum[i][1] = 0;
    int f8 = 1 << 8, f16 = 1 << 16, f24 = 1 << 24;                          // weights of the value bytes: factors of wide multiply-adds
    asm volatile("" : "+r"(f8), "+r"(f16), "+r"(f24));
    int4 v[8];                                                              // keys 8t .. 8t + 7 (steps 4t + i and 16 + 4t + i), dimensions 4g .. of 32
    auto value_rows = [&](int tile, int ch) {
        const int row = tile * AC_TILE + 8 * t;
        const int32_t *at = vc + (long long)row * HD + 4 * g + 32 * ch;
        if (tile + 1 < n_tiles) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = ac_load(at + i * HD);
        } else {                                                            // rows past the last read as it
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = ac_load(at + (long long)(min(row + i, last) - row) * HD);
        }
    };
    if (mine > 0) value_rows(first + warp, 0);
    j = 0;
    for (int tile = first + warp; tile < end; tile += AC_WARPS, j++) {
        ahead(mine + j + AC_AHEAD);
        const int4 *e4 = reinterpret_cast<const int4 *>(off + g * stride + (tile - first) * AC_TILE + 8 * t);
        const int4 lo4 = e4[0], hi4 = e4[1];
        uint32_t p[8] = {(uint32_t)lo4.x, (uint32_t)lo4.y, (uint32_t)lo4.z, (uint32_t)lo4.w, (uint32_t)hi4.x, (uint32_t)hi4.y, (uint32_t)hi4.z, (uint32_t)hi4.w};
        uint32_t any = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            p[i] = quotient(p[i]);
            any |= p[i];
        }
        uint32_t P0[4], P1[4];
        ac_bytes(p[0], p[1], p[2], p[3], P0); ac_bytes(p[4], p[5], p[6], p[7], P1);
        const bool third = __any_sync(0xffffffffu, (any >> 16) != 0);
#pragma unroll
        for (int ch = 0; ch < HD / 32; ch++) {
            uint32_t B0[4][4], B1[4][4];                                    // [step][byte]: column c of step n is dimension 32 ch + 4 c + n
            ac_bytes(v[0].x, v[1].x, v[2].x, v[3].x, B0[0]); ac_bytes(v[4].x, v[5].x, v[6].x, v[7].x, B1[0]);
            ac_bytes(v[0].y, v[1].y, v[2].y, v[3].y, B0[1]); ac_bytes(v[4].y, v[5].y, v[6].y, v[7].y, B1[1]);
            ac_bytes(v[0].z, v[1].z, v[2].z, v[3].z, B0[2]); ac_bytes(v[4].z, v[5].z, v[6].z, v[7].z, B1[2]);
            ac_bytes(v[0].w, v[1].w, v[2].w, v[3].w, B0[3]); ac_bytes(v[4].w, v[5].w, v[6].w, v[7].w, B1[3]);
            if (ch + 1 < HD / 32) value_rows(tile, ch + 1);
            else value_rows(min(tile + AC_WARPS, end - 1), 0);
#pragma unroll
            for (int n = 0; n < 4; n++) {
                int u[4][2];
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    int c[4];
                    if (b < 3) ac_mma_first<false>(c, P0[0], P0[1], P1[0], P1[1], B0[n][b], B1[n][b]);
                    else ac_mma_first<true>(c, P0[0], P0[1], P1[0], P1[1], B0[n][b], B1[n][b]);
                    u[b][0] = c[2] * 256 + c[0]; u[b][1] = c[3] * 256 + c[1];
                }
#pragma unroll
                for (int i = 0; i < 2; i++)
                    sum[4 * ch + n][i] += (long long)u[0][i] + (long long)u[1][i] * f8 + (long long)u[2][i] * f16 + (long long)u[3][i] * f24;
                if (third) {                                                // a probability of 2^16 and more (2^fa at most)
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        int c[4];
                        if (b < 3) ac_mma_first<false>(c, P0[2], 0u, P1[2], 0u, B0[n][b], B1[n][b]);
                        else ac_mma_first<true>(c, P0[2], 0u, P1[2], 0u, B0[n][b], B1[n][b]);
                        sum[4 * ch + n][0] += (long long)c[0] << (16 + 8 * b); sum[4 * ch + n][1] += (long long)c[1] << (16 + 8 * b);
                    }
                }
            }
        }
    }
    // ---- the warps' sums over scores and queries, then one CTA's, then the cluster's: a CTA reads out its share of the heads ----------
    __syncthreads();
    unsigned long long *warp_sum = reinterpret_cast<unsigned long long *>(ac_sm) + (size_t)warp * AC_HEADS * HD;           // [8][HD]
#pragma unroll
    for (int ch = 0; ch < HD / 32; ch++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            longlong2 *to = reinterpret_cast<longlong2 *>(warp_sum + g * HD + 32 * ch + 8 * t + 4 * i);
            to[0] = make_longlong2(sum[4 * ch][i], sum[4 * ch + 1][i]); to[1] = make_longlong2(sum[4 * ch + 2][i], sum[4 * ch + 3][i]);
        }
    __syncthreads();
    longlong2 *cta_sum = reinterpret_cast<longlong2 *>(ac_sm);
    for (int i = tid; i < AC_HEADS * HD / 2; i += AC_THREADS) {
        longlong2 v = cta_sum[i];
#pragma unroll
        for (int w = 1; w < AC_WARPS; w++) {
            const longlong2 o = cta_sum[w * AC_HEADS * HD / 2 + i];
            v.x += o.x; v.y += o.y;
        }
        cta_sum[i] = v;
    }
    cluster.sync();
    const int quads = rep * HD / 4, share = (quads + n_c - 1) / n_c, q_end = min(quads, (rank + 1) * share);
    int64_t *out = a.out + (long long)seq * a.H * HD + (long long)kv * rep * HD;
    for (int q = rank * share + tid; q < q_end; q += AC_THREADS) {          // four consecutive outputs per thread and turn
        long long y[4] = {0, 0, 0, 0};
        for (int r = 0; r < n_c; r++) {
            const longlong2 *src = cluster.map_shared_rank(cta_sum, r) + 2 * q;
            const longlong2 v0 = src[0], v1 = src[1];
            y[0] += v0.x; y[1] += v0.y; y[2] += v1.x; y[3] += v1.y;
        }
#pragma unroll
        for (int e = 0; e < 4; e++) out[4 * q + e] = y[e] >> a.fa;
    }
    cluster.sync();                                                         // nobody leaves while its sums are read
}

template <int HD, bool SHORT>
cudaError_t launch_cluster(const AttnArgs &a_in, int n_c, int tiles, cudaStream_t s) {
    AttnArgs a = a_in;
    a.chunk = tiles;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attn_cluster_kernel<HD, SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ac_smem<HD>(AC_MAX_TILES));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_cluster_kernel<HD, SHORT>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_c, (unsigned)a.Hkv, (unsigned)std::max(1, a.batch)); cfg.blockDim = dim3(AC_THREADS); cfg.stream = s;
    cfg.dynamicSmemBytes = ac_smem<HD>(tiles);
    cudaLaunchAttribute attr[2];
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // the kernel begins with pdl_enter()
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)n_c; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, attn_cluster_kernel<HD, SHORT>, a);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// Shapes: head dimensions 64 and 128, at most eight query heads per KV head, probabilities within three bytes, cache rows that 16-byte
// loads can start on.  a.pos is the position or its upper bound.
bool attn_cluster_plan(const AttnArgs &a, int &n_c, int &tiles) {
    if ((a.hd != 64 && a.hd != 128) || a.H / a.Hkv > AC_HEADS || a.fa > 23 || a.Hkv > 65535 || a.batch > 65535) return false;
    if ((reinterpret_cast<uintptr_t>(a.kcache) | reinterpret_cast<uintptr_t>(a.vcache)) & 15 || (a.seq_stride & 3)) return false;
    long long n_keys = a.pos + 1;
    if (a.window > 0 && n_keys > a.window) n_keys = a.window;
    const long long nt = (n_keys + AC_TILE - 1) / AC_TILE, pairs = (long long)a.Hkv * std::max(1, a.batch);
    if (nt > (long long)AC_MAX_TILES * AC_MAX_CLUSTER) return false;
    const int least = (int)((nt + AC_MAX_TILES - 1) / AC_MAX_TILES), most = (int)std::min<long long>(AC_MAX_CLUSTER, (nt + AC_WARPS - 1) / AC_WARPS);
    // as few rounds of a warp per CTA as the cluster allows; with two CTAs per SM and more at hand, the cluster whose rounds are fullest
    long long cost = 0;
    n_c = 0;
    for (int c = std::max(1, least); c <= std::max(1, std::max(least, most)); c++) {
        const long long rounds = ((nt + c - 1) / c + AC_WARPS - 1) / AC_WARPS, waves = (pairs * c + 2 * 148 - 1) / (2 * 148);
        const long long now = waves * (rounds + 3);                        // a CTA's start, exchanges and read-out cost about three rounds
        if (n_c == 0 || now < cost) { n_c = c; cost = now; }
    }
    tiles = (int)((nt + n_c - 1) / n_c);
    return true;
}

cudaError_t launch_attn_cluster(const AttnArgs &a, int n_c, int tiles, cudaStream_t s) {
    if (a.fa <= 16) return a.hd == 128 ? launch_cluster<128, true>(a, n_c, tiles, s) : launch_cluster<64, true>(a, n_c, tiles, s);
    return a.hd == 128 ? launch_cluster<128, false>(a, n_c, tiles, s) : launch_cluster<64, false>(a, n_c, tiles, s);
}

}  // namespace iie
