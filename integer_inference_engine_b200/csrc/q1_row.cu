// Q1_0 products of a single row (contract and unit layout: q1.cu).
//
// The row comes as int64 values, is RMS-normalised first where asked, and is split into its eight balanced digits by every CTA for
// itself, so that a product is one launch.  One CTA per SM walks 16-row tiles; warp w holds the digits of two 128-value blocks as
// MMA fragments and multiplies the two weight units of every tile with them.  Tiles come in groups of four by bulk copies into a ring.  The ring is filled before the wait for the preceding kernel of the stream, so the weights are on
// their way while that kernel still runs.  Rows longer than 32 blocks are cut into parts of at most 32 that add to the output.
//
// What bounds it: after the wait, the chain row load -> root -> digits -> fragments (about 2.5 us), then the multiplies, about 125
// instructions per two units of which 8 are MMAs; the weights arrive meanwhile.
#include "kernels.h"
#include "mma_items.cuh"
#include "norm.cuh"

#include <algorithm>
#include <type_traits>

namespace iie {

namespace {

constexpr int RW_WARPS = 16, RW_THREADS = RW_WARPS * 32;
constexpr int RW_BLOCKS = 2 * RW_WARPS;           // 128-value blocks of a part
constexpr int RW_VALUES = RW_BLOCKS * 128;
constexpr int RW_PLANE = RW_VALUES + 32;          // bytes of a digit plane: the eight planes of a fragment read start on different banks
constexpr int RW_GROUP = 4;                       // tiles between two reductions over the warps
constexpr int RW_COL = 20;                        // 8-byte words of a column of partial sums: sixteen rows and padding, so that half a
                                                  // warp writes (and reads) different banks
constexpr int RW_RING = 3;                         // groups the ring holds at most
constexpr unsigned RW_POLLS = 1u << 22;           // polls before a wait gives up and raises flag bit 3
constexpr size_t RW_PART_BYTES = (size_t)2 * RW_GROUP * 32 * RW_COL * 8;
constexpr size_t RW_HEAD_BYTES = (8 * (size_t)RW_PLANE > RW_PART_BYTES ? 8 * (size_t)RW_PLANE : RW_PART_BYTES);   // planes, then partial sums
static_assert(RW_HEAD_BYTES % 128 == 0, "ring slots stay aligned");

struct Q1RowArgs {
    const uint8_t *units[Q1_MAX_PARTS];           // matrices of the same row length
    int64_t *out[Q1_MAX_PARTS];
    const int64_t *add[Q1_MAX_PARTS];             // nullable: added to the product (may be `out`)
    long long out_f[Q1_MAX_PARTS];
    int tile_end[Q1_MAX_PARTS];                   // tiles up to and with that matrix
    int n_mats, tiles;                            // tiles of all matrices
    int nb, parts, part_blocks, per_part;         // blocks of the row, its parts, blocks of a part, CTAs of a part
    int depth, sh, small_scales;
    const int64_t *x, *gain;                      // the row; gain (nullable) where it is normalised
    int norm, frac;
    unsigned long long eps;
    int64_t log2e, clip;                          // SWIGLU
    int *flags;
};

__device__ __forceinline__ uint32_t rw_s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool rw_wait(uint32_t bar, uint32_t parity) {
    for (unsigned it = 0; it < RW_POLLS; it++) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// D(16x8,s32) = A(16x32,u8,row) * B(32x8,s8,col): the first step of a sum
__device__ __forceinline__ void rw_mma_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// Sums over the 128 values of a block of the set bits' values, for two units at once, times a factor of two: a lane ends with that
// of row g + 8 (t & 1) of unit t >> 1.  The columns of the MMA are the digits.  A register of weight bits is one AND behind a left
// shift (a multiplication, so that the logic unit, which bounds the walk over the tiles, has the ANDs alone): bits 6 and 7 of every
// byte stand for the rows g and g + 8, which doubles the latter (the digits' weights double the others).  Two exchanges bring the
// digits of a lane's row and unit together; with four digits in use (NARROW) every second column is zero and stays out.
// NARROW: 128 times the sums; otherwise, where the factor could carry into the wrapped product, twice them.
struct RowFold {
    int f[4];                                     // weights of the digits that this lane, lane xor 1, xor 2 and xor 3 hold
    bool second, odd;
    __device__ __forceinline__ explicit RowFold(int t) : second(t >= 2), odd(t & 1) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            f[k] = (odd ? 1 : 2) << (8 * (t ^ k));
            asm volatile("" : "+r"(f[k]));        // a factor, one wide multiply-add each: known as a power of two it would be a 64-bit shift
        }
    }
    __device__ __forceinline__ int64_t operator()(int a0, int a1, int b0, int b1) const {      // units a, b; rows g, g + 8
        const int k0 = second ? b0 : a0, k1 = second ? b1 : a1;
        const int o0 = __shfl_xor_sync(0xffffffffu, second ? a0 : b0, 2), o1 = __shfl_xor_sync(0xffffffffu, second ? a1 : b1, 2);
        const int own = odd ? k1 : k0, far = odd ? o1 : o0;
        const int near = __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 1), last = __shfl_xor_sync(0xffffffffu, odd ? o0 : o1, 1);
        return (int64_t)own * f[0] + (int64_t)near * f[1] + (int64_t)far * f[2] + (int64_t)last * f[3];
    }
};
template <bool NARROW>
__device__ __forceinline__ uint64_t rw_unit_sums(const uint2 (&w)[2], const uint32_t (&bf)[2][8], const RowFold &fold) {
    int c[2][4];
#pragma unroll
    for (int m = 0; m < 4; m++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t raw = (m >> 1) ? w[u].y : w[u].x, high = raw * ((m & 1) ? 1u : 16u), low = raw * ((m & 1) ? 4u : 64u);
            const uint32_t a0 = low & 0x40404040u, a1 = low & 0x80808080u, a2 = high & 0x40404040u, a3 = high & 0x80808080u;
            if (m == 0) rw_mma_first(c[u], a0, a1, a2, a3, bf[u][0], bf[u][1]);
            else mma_u8s8_k32(c[u], a0, a1, a2, a3, bf[u][2 * m], bf[u][2 * m + 1]);
        }
    if (!NARROW) {
#pragma unroll
        for (int u = 0; u < 2; u++) { c[u][0] >>= 6; c[u][1] >>= 6; c[u][2] >>= 6; c[u][3] >>= 6; }
    }
    uint64_t v = (uint64_t)fold(c[0][0], c[0][2], c[1][0], c[1][2]);
    if (!NARROW) v += (uint64_t)fold(c[0][1], c[0][3], c[1][1], c[1][3]) << 32;      // columns 2t + 1: digits four further up
    return v;
}

// SWIGLU: two matrices of the same rows, groups of their tiles taken alternately; out[0] = ((silu(product 0)) * product 1) >> frac
template <typename DT, bool SWIGLU, bool LATE>
__global__ void __launch_bounds__(RW_THREADS, 2) q1_row_kernel(const Q1RowArgs a) {
    constexpr int US = 256 + 16 * (int)sizeof(DT);
    extern __shared__ __align__(128) uint8_t rw_sm[];
    __shared__ __align__(8) uint64_t s_bars[RW_RING];
    __shared__ uint64_t s_lo[RW_WARPS], s_hi[RW_WARPS], s_total[RW_BLOCKS];
    __shared__ uint32_t s_bits[RW_WARPS];
    __shared__ int s_dead;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int part = blockIdx.x / a.per_part, seat = blockIdx.x - part * a.per_part;
    const int b0 = part * a.part_blocks, blocks = min(a.part_blocks, a.nb - b0);
    const int units = SWIGLU ? a.tiles >> 1 : a.tiles;                    // tiles, or pairs of them
    const int lo = (int)((long long)units * seat / a.per_part), run = (int)((long long)units * (seat + 1) / a.per_part) - lo;
    const int groups = ((run + RW_GROUP - 1) / RW_GROUP) << (SWIGLU ? 1 : 0);
    uint8_t *ring = rw_sm + RW_HEAD_BYTES;
    const uint32_t bars = rw_s32(s_bars), tile_bytes = (uint32_t)(blocks * US), tile_stride = (uint32_t)(((a.part_blocks + 1) & ~1) * US);
    // tiles of this CTA's run in groups; SWIGLU: a group of the first matrix, then the same tiles of the second
    auto group_tiles = [&](int q) { return min(RW_GROUP, run - RW_GROUP * (SWIGLU ? q >> 1 : q)); };
    auto place = [&](int q, int i, int &mat, int &tile) {
        const int v = lo + RW_GROUP * (SWIGLU ? q >> 1 : q) + i;
        mat = SWIGLU ? q & 1 : 0; tile = v;
        if (!SWIGLU) {
#pragma unroll
            for (int m = 0; m + 1 < Q1_MAX_PARTS; m++)
                if (m + 1 < a.n_mats && v >= a.tile_end[m]) { mat = m + 1; tile = v - a.tile_end[m]; }
        }
    };
    // lane i < tiles of the group: tile i of group q into place s of the ring
    auto request = [&](int q, int s) {
        const int n = group_tiles(q);
        const uint32_t bar = bars + 8 * s;
        if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n * tile_bytes) : "memory");
        __syncwarp();
        if (lane < n) {
            int mat, tile;
            place(q, lane, mat, tile);
            const uint8_t *base = mat == 0 ? a.units[0] : mat == 1 ? a.units[1] : a.units[2];
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(rw_s32(ring) + (s * RW_GROUP + lane) * tile_stride), "l"(base + ((long long)tile * a.nb + b0) * US),
                           "r"(tile_bytes), "r"(bar) : "memory");
        }
    };
    if (warp == 0) {
        if (lane < a.depth) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * lane));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (lane == 0) s_dead = 0;
        __syncwarp();
        for (int q = 0; q < min(a.depth, groups); q++) request(q, q);
    }
    // The gain is read ahead of the wait where the kernel in front does not write it, else (LATE) brought to the cache here and read behind
    // the wait.  Forms of their own: one form for both, or the late one alone, cost 0.4 us of a product (q1 decode 1600 against 1632 us).
    const int K = a.nb * 128, pk = blocks * 128;
    int64_t gv[2][4];
    uint64_t gm = 1;
    auto read_gain = [&]() {
        if (a.norm && a.gain) {
            gm = 0;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int i = 4 * (tid + q * RW_THREADS);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    gv[q][e] = i < pk ? (LATE ? a.gain[b0 * 128 + i + e] : __ldg(a.gain + b0 * 128 + i + e)) : 0;
                    gm |= uabs64(gv[q][e]);
                }
            }
            if (a.parts > 1) for (int i = tid; i < K; i += RW_THREADS) gm |= uabs64(LATE ? a.gain[i] : __ldg(a.gain + i));
        } else {
#pragma unroll
            for (int q = 0; q < 2; q++) { gv[q][0] = gv[q][1] = gv[q][2] = gv[q][3] = 1; }
        }
    };
    if (!LATE) read_gain();
    else if (a.norm && a.gain) for (int i = 16 * tid; i < pk; i += 16 * RW_THREADS) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.gain + b0 * 128 + i));
    // behind this wait everything before the preceding kernel has finished, too: each kernel starts its dependents behind its own wait
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");

    // ---- this part of the row: normalise, split into digit planes -----------------------------------------------------------
    int64_t x[2][4];
    uint64_t all = 0;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int i = 4 * (tid + q * RW_THREADS);
        longlong2 v0 = make_longlong2(0, 0), v1 = v0;
        if (i < pk) {
            const int64_t *src = a.x + (long long)b0 * 128 + i;
            v0 = *reinterpret_cast<const longlong2 *>(src); v1 = *reinterpret_cast<const longlong2 *>(src + 2);
        }
        x[q][0] = v0.x; x[q][1] = v0.y; x[q][2] = v1.x; x[q][3] = v1.y;
    }
    if (LATE) read_gain();
#pragma unroll
    for (int q = 0; q < 2; q++) all |= uabs64(x[q][0]) | uabs64(x[q][1]) | uabs64(x[q][2]) | uabs64(x[q][3]);
    bool bad = false, narrow = (all >> 30) == 0;                          // four digits hold every value
    if (a.norm) {
        u128 ssq = 0;
        auto take = [&](int64_t v) { const uint64_t m = uabs64(v); ssq += (u128)m * m; all |= m; };
        if ((all >> 31) == 0) {
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int e = 0; e < 4; e++) ssq += (uint64_t)((int64_t)(int)x[q][e] * (int)x[q][e]);
        } else {
#pragma unroll
            for (int q = 0; q < 2; q++) { take(x[q][0]); take(x[q][1]); take(x[q][2]); take(x[q][3]); }
        }
        if (a.parts > 1)
            for (int i = tid; i < K; i += RW_THREADS) if (i < b0 * 128 || i >= b0 * 128 + pk) take(a.x[i]);
        // (an |x| of exactly 2^57 may be flagged beyond with other bits set: checked exactly below)
        uint32_t xb = __reduce_max_sync(0xffffffffu, (uint32_t)(64 - __clzll((long long)all)));
        uint32_t gb = __reduce_max_sync(0xffffffffu, (uint32_t)(64 - __clzll((long long)gm)));
        ssq = warp_sum128(ssq);
        if (lane == 0) { s_lo[warp] = (uint64_t)ssq; s_hi[warp] = (uint64_t)(ssq >> 64); s_bits[warp] = xb | gb << 8; }
        __syncthreads();
        ssq = warp_sum128(lane < RW_WARPS ? ((u128)s_hi[lane] << 64) | s_lo[lane] : (u128)0);
        const uint32_t bits = lane < RW_WARPS ? s_bits[lane] : 0;
        xb = __reduce_max_sync(0xffffffffu, bits & 0xFF); gb = __reduce_max_sync(0xffffffffu, bits >> 8);
        bool beyond = K > 8192;
        if (xb >= 58)                                                     // rare: |x| beyond 2^57 exactly?
            for (int i = 0; i < K; i += 32) beyond = __any_sync(0xffffffffu, beyond || (i + lane < K && uabs64(a.x[i + lane]) > (1ULL << 57)));
        const NormRow n(ssq, (int)xb, (int)gb, beyond, K, a.eps, a.frac, a.gain != nullptr);
        bad = n.refused;                                                  // the products of zeros are stored, and the flag
        narrow = n.fast || n.refused;
        if (narrow) {
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int e = 0; e < 4; e++) x[q][e] = n.refused ? 0 : n.fast_value((int)x[q][e], (int)gv[q][e]);
        } else {                                                          // the general form, through shared memory to keep it short
            const uint64_t inv = n.rms < (1ULL << 62) ? recip_below(n.rms) : 0, gmax = a.gain ? warp_gain_max(a.gain, K) : 0;
            int64_t *own = reinterpret_cast<int64_t *>(rw_sm);
#pragma unroll 1
            for (int k = 0; k < 8; k++) {
                const int i = 4 * (tid + (k >> 2) * RW_THREADS) + (k & 3), at = b0 * 128 + i;
                own[tid * 8 + k] = i < pk ? norm_value(a.x[at], n.rms, inv, gmax, a.gain ? a.gain[at] : 0, a.gain != nullptr, a.frac, bad) : 0;
            }
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int e = 0; e < 4; e++) x[q][e] = own[tid * 8 + 4 * q + e];
            __syncthreads();
        }
    } else {
        narrow = __syncthreads_and(narrow);
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {                                         // a warp's four times 32 values are a block
        const uint64_t sum = (uint64_t)warp_sum64((uint64_t)x[q][0] + (uint64_t)x[q][1] + (uint64_t)x[q][2] + (uint64_t)x[q][3]);
        if (lane == 0) s_total[warp + RW_WARPS * q] = sum;
        uint32_t d[2][4];                                                 // [low, high word of the digits][element]
        if (narrow) {
#pragma unroll
            for (int e = 0; e < 4; e++) { d[0][e] = ((uint32_t)x[q][e] + 0x80808080u) ^ 0x80808080u; d[1][e] = 0; }      // byte l: balanced digit l
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint64_t y = ((uint64_t)x[q][e] + 0x8080808080808080ULL) ^ 0x8080808080808080ULL;
                d[0][e] = (uint32_t)y; d[1][e] = (uint32_t)(y >> 32);
            }
        }
#pragma unroll
        for (int half = 0; half < 2; half++) {
            if (half && narrow) break;                                    // never read
            const uint32_t t0 = __byte_perm(d[half][0], d[half][1], 0x5140), t1 = __byte_perm(d[half][2], d[half][3], 0x5140);
            const uint32_t t2 = __byte_perm(d[half][0], d[half][1], 0x7362), t3 = __byte_perm(d[half][2], d[half][3], 0x7362);
            uint8_t *to = rw_sm + (size_t)(4 * half) * RW_PLANE + 4 * (tid + q * RW_THREADS);
            *reinterpret_cast<uint32_t *>(to) = __byte_perm(t0, t1, 0x5410);
            *reinterpret_cast<uint32_t *>(to + RW_PLANE) = __byte_perm(t0, t1, 0x7632);
            *reinterpret_cast<uint32_t *>(to + 2 * RW_PLANE) = __byte_perm(t2, t3, 0x5410);
            *reinterpret_cast<uint32_t *>(to + 3 * RW_PLANE) = __byte_perm(t2, t3, 0x7632);
        }
    }
    __syncthreads();
    uint32_t bf[2][8];
    {
        const int digit = col_limb(g);
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int m = 0; m < 4; m++) {
                uint2 v = make_uint2(0, 0);
                if (2 * warp + u < blocks && !(narrow && digit >= 4)) v = *reinterpret_cast<const uint2 *>(rw_sm + (size_t)digit * RW_PLANE + (2 * warp + u) * 128 + 32 * m + 8 * t);
                bf[u][2 * m] = v.x; bf[u][2 * m + 1] = v.y;
            }
    }
    __syncthreads();                                                      // the planes' space takes the partial sums from here on
    uint64_t *part_sums = reinterpret_cast<uint64_t *>(rw_sm);           // [2][RW_GROUP][32 shares][RW_COL]

    // ---- tiles: a warp's share of a tile's sixteen rows are two columns (one per unit) of the partial sums; behind every group the
    //      sixteen warps add the columns up, four rows of one tile each, eight lanes a row --------------------------------------
    uint64_t result = 0;                                                  // lane 4 o + r: row 4 (warp % 4) + r of tile warp / 4 of group 8 k + o
    const int end_i = warp >> 2, end_r = 4 * (warp & 3) + (lane & 3);
    auto finish = [&](int q0, int n_groups) {                             // groups q0 .. q0 + n_groups - 1
        const int q = q0 + (lane >> 2);
        int mat = 0, tile = 0;
        const bool live = (lane >> 2) < n_groups && end_i < group_tiles(q);
        place(q, end_i, mat, tile);
        const long long row = (long long)tile * 16 + end_r;
        if (SWIGLU) {
            const uint64_t up = __shfl_down_sync(0xffffffffu, result, 4);
            if (live && !(q & 1) && row < a.out_f[0]) {
                const int64_t gate = (int64_t)result, sg = sigmoid_fixed_c(gate, a.frac, a.log2e, a.clip);
                const int64_t silu = (int64_t)((uint64_t)gate * (uint64_t)sg) >> a.frac;
                a.out[0][row] = (int64_t)((uint64_t)silu * up) >> a.frac;
            }
        } else if (live) {
            const long long rows = mat == 0 ? a.out_f[0] : mat == 1 ? a.out_f[1] : a.out_f[2];
            int64_t *out = mat == 0 ? a.out[0] : mat == 1 ? a.out[1] : a.out[2];
            const int64_t *add = mat == 0 ? a.add[0] : mat == 1 ? a.add[1] : a.add[2];
            if (row < rows) {
                if (a.parts > 1) atomicAdd(reinterpret_cast<unsigned long long *>(out + row), (unsigned long long)result);
                else out[row] = (int64_t)(result + (add ? (uint64_t)add[row] : 0));
            }
        }
    };
    bool dead = false;
    auto walk = [&](auto tag) {
        constexpr bool NARROW = decltype(tag)::value;
        const RowFold fold(t);
        const int column = (2 * warp + (t >> 1)) * RW_COL + g + 8 * (t & 1);
        // blocks beyond the part have no digits, so whatever units stand in for theirs add nothing
        const int first = min(2 * warp, ((a.part_blocks + 1) & ~1) - 2);
        const uint64_t total = s_total[2 * warp + (t >> 1)] * (NARROW ? 64 : 1);
        const int sh = a.sh + (NARROW ? 6 : 0);
        int s = 0, asked = min(a.depth, groups);                          // behind a failure nothing more is asked for, and only that awaited
        uint32_t parity = 0;
        for (int q = 0; q < groups; q++) {
            const int n = group_tiles(q);
            uint64_t *sums = part_sums + (size_t)(q & 1) * RW_GROUP * 32 * RW_COL;
            if (q < asked && !__all_sync(0xffffffffu, rw_wait(bars + 8 * s, parity))) { dead = true; s_dead = 1; }
            const uint8_t *unit = ring + (size_t)(s * RW_GROUP) * tile_stride + first * US;
            uint64_t *to = sums + column;
#pragma unroll 1
            for (int i = 0; i < n; i++) {
                const uint2 w[2] = {*reinterpret_cast<const uint2 *>(unit + lane * 8), *reinterpret_cast<const uint2 *>(unit + US + lane * 8)};
                const int64_t sc = (int64_t)*(reinterpret_cast<const DT *>(unit + (t >> 1) * US + 256) + g + 8 * (t & 1));
                *to = (uint64_t)((int64_t)((rw_unit_sums<NARROW>(w, bf, fold) - total) * (uint64_t)sc) >> sh);
                unit += tile_stride; to += 32 * RW_COL;
            }
            __syncthreads();                                              // the group has been read; the other half of the sums is free
            if (!dead && asked < groups) { if (warp == 0) request(asked, s); asked++; }
            if (++s == a.depth) { s = 0; parity ^= 1; }
            if (end_i < n) {
                const uint64_t *from = sums + (end_i * 32 + (lane >> 2)) * RW_COL + end_r;
                uint64_t v = from[0] + from[8 * RW_COL] + from[16 * RW_COL] + from[24 * RW_COL];
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                v += __shfl_xor_sync(0xffffffffu, v, 8);
                v += __shfl_xor_sync(0xffffffffu, v, 16);
                if ((lane >> 2) == (q & 7)) result = v;
            }
            if (s_dead) continue;                                         // a copy never arrived: nothing is stored from here on
            if ((q & 7) == 7 || q + 1 == groups) finish(q & ~7, (q & 7) + 1);
        }
    };
    // (products of narrow values with scales below 2^20 keep the factor of 64 within 64 bits)
    if (narrow && a.small_scales) walk(std::true_type()); else walk(std::false_type());
    if (dead && lane == 0) atomicOr(a.flags, 8);
    if (bad) atomicOr(a.flags, 2);
}

__global__ void q1_row_init_kernel(int64_t *out, const int64_t *add, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = add ? add[i] : 0;
}

template <typename DT, bool SWIGLU, bool LATE>
cudaError_t launch_row(const Q1RowArgs &a, cudaStream_t s) {
    const int run = (a.tiles / (SWIGLU ? 2 : 1) + a.per_part - 1) / a.per_part, groups = (run + RW_GROUP - 1) / RW_GROUP * (SWIGLU ? 2 : 1);
    Q1RowArgs b = a;
    // two groups ahead leave room for the next kernel's CTAs beside these; a long run (an output matrix) takes three
    b.depth = groups >= 8 ? RW_RING : std::min(groups, 2);
    const size_t tile = (size_t)((b.part_blocks + 1) & ~1) * (256 + 16 * sizeof(DT));
    // tiles of the ring: a run that fits in it whole takes no more than its tiles
    const size_t slots = groups <= b.depth ? (size_t)(b.depth - 1) * RW_GROUP + (SWIGLU ? std::min(run, RW_GROUP) : run - (groups - 1) * RW_GROUP) : (size_t)b.depth * RW_GROUP;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(q1_row_kernel<DT, SWIGLU, LATE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(RW_HEAD_BYTES + (size_t)RW_RING * RW_GROUP * RW_BLOCKS * (256 + 16 * sizeof(DT))));
        // all of the SM's memory as shared memory: otherwise the next kernel's CTAs do not fit beside these and start behind them, two to an SM
        if (e == cudaSuccess) e = cudaFuncSetAttribute(q1_row_kernel<DT, SWIGLU, LATE>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(b.parts * b.per_part)); cfg.blockDim = dim3(RW_THREADS); cfg.stream = s;
    cfg.dynamicSmemBytes = RW_HEAD_BYTES + slots * tile;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, q1_row_kernel<DT, SWIGLU, LATE>, b);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// Parts: as few as hold the row, of the same size; the SMs are shared out among them, so that a CTA stays within one part
// (12288 values: 3 x 49 CTAs of 5 to 6 tiles; splitting a row also divides the row's load and digits among the CTAs).
cudaError_t launch_q1_row(const Q1Part *mats, int n, bool sc32, long long nb, const Q1RowInput &in, bool swiglu, long long frac, cudaStream_t s) {
    if (n < 1 || n > Q1_MAX_PARTS || nb <= 0 || nb > (1 << 20) || !in.x || (swiglu && (n != 2 || mats[0].out_f != mats[1].out_f))) return cudaErrorInvalidValue;
    Q1RowArgs a = {};
    for (int i = 0; i < n; i++) {
        a.units[i] = mats[i].units; a.out[i] = mats[i].out; a.add[i] = mats[i].add; a.out_f[i] = mats[i].out_f;
        const long long tiles = a.tiles + (mats[i].out_f + 15) / 16;
        if (tiles > (1 << 28)) return cudaErrorInvalidValue;
        a.tiles = (int)tiles; a.tile_end[i] = a.tiles;
    }
    a.small_scales = frac <= 57;
    for (int i = 0; i < n; i++) if (mats[i].max_scale >= (1u << 20)) a.small_scales = 0;
    a.n_mats = n; a.nb = (int)nb;
    a.parts = (int)((nb + RW_BLOCKS - 1) / RW_BLOCKS);
    a.part_blocks = (int)((nb + a.parts - 1) / a.parts);
    a.parts = (int)((nb + a.part_blocks - 1) / a.part_blocks);
    if (swiglu && a.parts > 1) return cudaErrorNotSupported;             // the two products are complete in no CTA
    a.per_part = std::max(1, std::min(148 / a.parts, swiglu ? a.tiles / 2 : a.tiles));
    a.sh = frac <= 0 ? 0 : (frac >= 63 ? 63 : (int)frac);
    a.x = in.x; a.gain = in.gain; a.norm = in.norm ? 1 : 0; a.frac = (int)frac; a.eps = in.eps;
    if (swiglu) { a.log2e = sigmoid_log2e((int)frac); a.clip = sigmoid_clip((int)frac); }
    a.flags = shared_flag_word();
    if (!a.flags) return cudaErrorInvalidValue;
    for (int i = 0; a.parts > 1 && i < n; i++)
        if (mats[i].add != mats[i].out) {
            q1_row_init_kernel<<<(unsigned)((mats[i].out_f + 255) / 256), 256, 0, s>>>(mats[i].out, mats[i].add, mats[i].out_f);
            note_launch();
        }
    const bool late = in.norm && in.gain && !in.gain_ahead;
    if (swiglu && late) return cudaErrorNotSupported;                    // (no caller has that)
    if (swiglu) return sc32 ? launch_row<int, true, false>(a, s) : launch_row<long long, true, false>(a, s);
    if (late) return sc32 ? launch_row<int, false, true>(a, s) : launch_row<long long, false, true>(a, s);
    return sc32 ? launch_row<int, false, false>(a, s) : launch_row<long long, false, false>(a, s);
}

}  // namespace iie
