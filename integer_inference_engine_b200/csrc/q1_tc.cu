// Q1_0 products of two tokens and more on the 5th-generation tensor cores (tcgen05 kind::i8).
//
// out[t, o] = sum_b floor((sum_{i<128} s_i x[t, 128 b + i]) * scale[o, b] / 2^frac)   (mod 2^64), see q1.cu.
//
// A CTA multiplies tiles of 128 weight rows (MMA M, TMEM lanes) x NT tokens, one 128-weight block at a time:
//   A = the block's signs as bytes +1 / -1 (128 rows x 128 bytes, 128-byte swizzle), expanded from the registered bit words;
//   B = the digit planes of the NT tokens (fetched by TMA), stacked along N: the np planes in use make ONE MMA of
//       N = np * NT columns per K step, so the expanded signs are read once per K step and not once per plane;
//   D = np accumulators of NT columns, in two or four TMEM buffers.
// The floor is per block, so every block's accumulators are read out: acc = sum_l 256^l D_l, acc * scale, shift, add.  With
// three planes (-8421504 <= x <= 8355711, what a normalised row has) |acc| stays below 128 * 8421504 < 2^31 and the read-out is one
// 32 x 32 -> 64 multiplication; more planes take 64-bit sums.
//
// Roles: eight or sixteen read-out warps (lane = row, a share of the tokens each), four expanding warps, one warp each for the
// MMAs, the planes' TMA loads and the bulk copies of the registered units (bit words and scales of eight blocks per copy).
// What bounds it: the integer instructions of the read-out (about 8 per row, token and block) and the hand-overs of a block,
// about 1600 clocks per block of a 128 x 64 tile of which the MMAs (4 x N = 192) take 480.  12288 x 4096 at 512 tokens: 162 us
// (546 us with one MMA per plane, 0 / 1 operands, 64-bit sums for every digit count and one accumulator buffer); at 6 tokens
// 14 us (370 us with warp-level MMAs), 4096 x 4096 at 6 tokens 8.6 us (123).  Up to eight tokens a tile of eight halves the read-out:
// a step of six sequences 1504 -> 1465 us (the hand-overs of a block stay).
//
// Split of the work: with at least four tiles per SM each CTA walks whole tiles.  With fewer, the (tile, block) pairs of all
// tiles are dealt out evenly (a CTA then owns a contiguous run of blocks that may begin and end inside a tile) and the shares
// of a tile are added with atomics to the residual row in place or to zeros that the kernel in front has written.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "common.cuh"

namespace iie {

namespace {

constexpr int QC_EXPAND = 4;
// read-out warps: sixteen where 64 tokens have to be read out per block, eight where less work would not pay for their waits
__host__ __device__ constexpr int qc_read_warps(int nt) { return nt == 64 ? 16 : 8; }
__host__ __device__ constexpr int qc_threads(int nt) { return (qc_read_warps(nt) + QC_EXPAND + 3) * 32; }
constexpr int QC_MAX_STAGES = 6, QC_RAW_SLOTS = 3, QC_CHUNK = 8;
constexpr int QC_A_BYTES = 128 * 128;
constexpr int QC_SMEM = 225 * 1024;
constexpr unsigned QC_WAIT_LIMIT = 1u << 17;

struct Q1TcArgs {
    Q1Part part[Q1_MAX_PARTS];
    int tile_end[Q1_MAX_PARTS];      // 128-row tiles of parts 0..p
    int n_parts, n_ttiles;           // token tiles of NT
    int nb;
    long long T;
    int sh;
    int narrow;                      // the scales are small enough for the three-plane read-out
    int split;                       // 0: whole tiles, CTA c takes tiles c, c + grid, ...; 1: blocks dealt out evenly
    long long n_tiles;
    const int *nl_dev;               // digit planes in use (planes at and above it are zero)
    int *flags;                      // bit 3 is raised when a wait ran out
};

__device__ __forceinline__ uint32_t qc_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// barriers by their shared-memory address
__device__ __forceinline__ void qc_init(uint32_t b, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n)); }
__device__ __forceinline__ void qc_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory"); }
__device__ __forceinline__ void qc_expect(uint32_t b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool qc_try(uint32_t b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(b), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __noinline__ bool qc_wait_slow(uint32_t b, uint32_t parity, volatile int *abort_flag) {      // bounded
    for (unsigned it = 0; it < QC_WAIT_LIMIT; it++) {
        uint32_t ok;                                               // asleep for up to 20 us at a time
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(b), "r"(parity), "r"(20000u) : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool qc_wait(uint32_t b, uint32_t parity, volatile int *abort_flag) {
    return qc_try(b, parity) || qc_wait_slow(b, parity, abort_flag);
}
__device__ __forceinline__ bool qc_wait_warp(uint32_t b, uint32_t parity, volatile int *abort_flag) {  // the whole warp, one answer
    if (__all_sync(0xffffffffu, qc_try(b, parity))) return true;
    return __all_sync(0xffffffffu, qc_wait_slow(b, parity, abort_flag));
}
// Position in a ring of slots: `pass` is the parity of the current lap.  (Stepped, not computed from a running index: a division
// by a run-time slot count in every role's loop cost more than the rest of a block.)
struct Ring {
    int slot = 0;
    uint32_t pass = 0;
    bool lapped = false;                                           // every slot has been used once
    __device__ __forceinline__ void step(int n) { if (++slot == n) { slot = 0; pass ^= 1; lapped = true; } }
};
__device__ __forceinline__ uint32_t qc_elect() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r;
}
__device__ __forceinline__ void qc_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void qc_commit(uint32_t b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(b) : "memory");
}
// K-major operand rows of 128 bytes, 128-byte swizzle, eight-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t qc_desc(uint32_t smem) {
    return (uint64_t)((smem >> 4) & 0x3FFF) | (1ULL << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ULL << 46) | (2ULL << 61);
}

// sum += (a * b) & {~0, keep}
__device__ __forceinline__ void qc_mul_add(uint32_t &slo, uint32_t &shi, int a, int b, uint32_t keep) {
    asm("{\n .reg .b64 v;\n .reg .b32 lo, hi;\n mul.wide.s32 v, %2, %3;\n mov.b64 {lo, hi}, v;\n"
        " and.b32 lo, lo, %4;\n add.cc.u32 %0, %0, lo;\n addc.u32 %1, %1, hi;\n}"
        : "+r"(slo), "+r"(shi) : "r"(a), "r"(b), "r"(keep));
}
__device__ __forceinline__ void qc_tmem_ld(uint32_t addr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// planes carried for `nl` digits in use: the read-out exists for these counts
__device__ __forceinline__ int qc_planes(int nl, bool narrow) { return nl <= 3 && narrow ? 3 : nl <= 4 ? 4 : nl <= 6 ? 6 : 8; }

template <int NT, typename DT>
__global__ void __launch_bounds__(qc_threads(NT), 1) q1_tc_kernel(const Q1TcArgs a, const __grid_constant__ CUtensorMap xmap) {
    constexpr int US = 256 + 16 * (int)sizeof(DT);
    constexpr int RAW_BYTES = 8 * QC_CHUNK * US;                   // eight 16-row sub-tiles x eight blocks
    constexpr int QC_READ = qc_read_warps(NT), QC_MMA_WARP = QC_READ + QC_EXPAND, QC_PLANE_WARP = QC_MMA_WARP + 1;
    constexpr int TPW = NT * 4 / QC_READ;                          // tokens of a read-out thread
    extern __shared__ __align__(1024) unsigned char qc_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(qc_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * QC_MAX_STAGES + 2 * 4 + 2 * QC_RAW_SLOTS];
    const uint32_t full_bar = qc_u32(bars), empty_bar = full_bar + 8 * QC_MAX_STAGES, acc_bar = empty_bar + 8 * QC_MAX_STAGES, free_bar = acc_bar + 8 * 4,
                   raw_full = free_bar + 8 * 4, raw_empty = raw_full + 8 * QC_RAW_SLOTS;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nb = a.nb;
    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < QC_MAX_STAGES; s++) { qc_init(full_bar + 8 * s, QC_EXPAND + 1); qc_init(empty_bar + 8 * s, 1); }
        for (int s = 0; s < 4; s++) { qc_init(acc_bar + 8 * s, 1); qc_init(free_bar + 8 * s, QC_READ); }
        for (int s = 0; s < QC_RAW_SLOTS; s++) { qc_init(raw_full + 8 * s, 1); qc_init(raw_empty + 8 * s, QC_READ); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == QC_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(qc_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    pdl_enter();                                                   // what stands above needs nothing of the kernel before
    const int np = qc_planes(max(1, min(8, *a.nl_dev)), a.narrow);           // uniform over the grid
    const int mp = NT == 8 && np == 3 ? 4 : np;                    // planes multiplied: an instruction takes whole sixteens of columns (the fourth plane is zero)
    const int cols = mp * NT;                                      // TMEM columns of one buffer
    const int nbuf = cols <= 128 ? 4 : cols <= 256 ? 2 : 1, buf_cols = 512 / nbuf;
    const int stage_bytes = QC_A_BYTES + cols * 128;
    const int stages = min(QC_MAX_STAGES, (QC_SMEM - 1024 - QC_RAW_SLOTS * RAW_BYTES) / stage_bytes);
    unsigned char *raw = smem + stages * stage_bytes;

    // this CTA's run of (tile, block) pairs: u in [u0, u1), tile = t0 + (u / nb) * tstep, block = u % nb
    long long u0, u1, t0, tstep;
    if (a.split) {
        const long long W = a.n_tiles * nb;
        u0 = W * blockIdx.x / gridDim.x; u1 = W * (blockIdx.x + 1) / gridDim.x;
        t0 = 0; tstep = 1;
    } else {
        u0 = 0; u1 = blockIdx.x < a.n_tiles ? (a.n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x * nb : 0;
        t0 = blockIdx.x; tstep = gridDim.x;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    // row tile rt -> its part and the tile's index in it
    auto locate = [&](long long tile, int &p, int &rt, int &tt) {
        rt = (int)(tile / a.n_ttiles); tt = (int)(tile - (long long)rt * a.n_ttiles);
        p = 0;
        while (p + 1 < a.n_parts && rt >= a.tile_end[p]) p++;
        if (p > 0) rt -= a.tile_end[p - 1];
    };

    if (warp < QC_READ) {
        // ================= read-out: TMEM lane = row of the tile ==============================================
        const int rowt = (warp & 3) * 32 + lane, cg = warp >> 2;
        const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int scale_off = (rowt >> 4) * (QC_CHUNK * US) + 256 + (rowt & 15) * (int)sizeof(DT);
        auto read_out = [&](auto np_c) {
            constexpr int NP = decltype(np_c)::value;
            const uint32_t keep = 0xFFFFFFFFu << a.sh;         // three planes: the shift is below 32
            constexpr int RT = 4, ROUNDS = TPW / RT;               // tokens of a round; the next round's values load under this one's sums
            constexpr bool AHEAD = NP <= 4;                        // (where the registers hold two rounds)
            unsigned long long sum[TPW]; uint32_t slo[TPW], shi[TPW];
#pragma unroll
            for (int j = 0; j < TPW; j++) { slo[j] = 0; shi[j] = 0; }
#pragma unroll
            for (int j = 0; j < TPW; j++) sum[j] = 0;
            Ring unit, buf;
            for (long long u = u0; u < u1;) {
                const long long tl = u / nb, tile = t0 + tl * tstep;
                const int b0 = (int)(u - tl * nb), b1 = (int)min((long long)nb, b0 + (u1 - u));
                bool ok = true;
                for (int b = b0; b < b1; b++) {
                    if (b == b0 || (b & (QC_CHUNK - 1)) == 0) {
                        ok = qc_wait_warp(raw_full + 8 * unit.slot, unit.pass, &s_abort);
                        if (!ok) break;
                    }
                    const DT sc = *reinterpret_cast<const DT *>(raw + unit.slot * RAW_BYTES + (b & (QC_CHUNK - 1)) * US + scale_off);
                    ok = qc_wait_warp(acc_bar + 8 * buf.slot, buf.pass, &s_abort);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t base = tlane + buf.slot * buf_cols + cg * TPW;
                    int r[AHEAD ? 2 : 1][NP][RT];
#pragma unroll
                    for (int l = 0; l < NP; l++) qc_tmem_ld(base + l * NT, r[0][l]);
#pragma unroll
                    for (int ro = 0; ro < ROUNDS; ro++) {
                        if (!AHEAD && ro > 0) {
#pragma unroll
                            for (int l = 0; l < NP; l++) qc_tmem_ld(base + l * NT + ro * RT, r[0][l]);
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (AHEAD && ro + 1 < ROUNDS) {
#pragma unroll
                            for (int l = 0; l < NP; l++) qc_tmem_ld(base + l * NT + (ro + 1) * RT, r[(ro + 1) & 1][l]);
                        }
                        if (ro + 1 == ROUNDS) {                                   // the buffer is free as soon as its last values have landed
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) qc_arrive(free_bar + 8 * buf.slot);
                        }
#pragma unroll
                        for (int j = 0; j < RT; j++) {
                            const auto &x = r[AHEAD ? ro & 1 : 0];
                            long long v;
                            if (NP == 3) {
                                // |acc| <= 1077952512, and the launcher has seen to it that no sum of products leaves 64 bits: the bits
                                // below the shift are dropped here (the floor), the shift itself is taken once per tile
                                const int acc = x[0][j] + x[1][j] * 256 + x[2][j] * 65536;
                                if (sizeof(DT) == 4) { qc_mul_add(slo[ro * RT + j], shi[ro * RT + j], acc, (int)sc, keep); continue; }
                                v = ((long long)acc * (long long)sc) & (long long)(0xFFFFFFFF00000000ULL | keep);
                            } else {
                                long long lo = (long long)x[0][j];
#pragma unroll
                                for (int l = 1; l < 4 && l < NP; l++) lo += (long long)x[l][j] * (long long)(1 << (8 * l));
                                unsigned long long P = (unsigned long long)lo;
                                if (NP > 4) {
                                    long long hi4 = (long long)x[NP > 4 ? 4 : 0][j];
#pragma unroll
                                    for (int l = 5; l < NP; l++) hi4 += (long long)x[l][j] * (long long)(1 << (8 * (l - 4)));
                                    P += (unsigned long long)hi4 << 32;
                                }
                                v = (long long)(P * (unsigned long long)(long long)sc) >> a.sh;
                            }
                            sum[ro * RT + j] += (unsigned long long)v;
                        }
                    }
                    buf.step(nbuf);
                    if (b + 1 == b1 || ((b + 1) & (QC_CHUNK - 1)) == 0) {
                        __syncwarp();
                        if (lane == 0) qc_arrive(raw_empty + 8 * unit.slot);
                        unit.step(QC_RAW_SLOTS);
                    }
                }
                if (!ok) break;
                u += b1 - b0;
                // ---- the tile's sums, or this CTA's share of them --------------------------------------------
                if (NP == 3) {
#pragma unroll
                    for (int j = 0; j < TPW; j++) {
                        if (sizeof(DT) == 4) { sum[j] = ((unsigned long long)shi[j] << 32) | slo[j]; slo[j] = 0; shi[j] = 0; }
                        sum[j] = (unsigned long long)((long long)sum[j] >> a.sh);
                    }
                }
                int p, rt, tt;
                locate(tile, p, rt, tt);
                const long long row = (long long)rt * 128 + rowt, out_f = a.part[p].out_f;
                if (row < out_f) {
                    int64_t *out = a.part[p].out;
                    const int64_t *add = a.part[p].add;
                    const bool whole = b1 - b0 == nb;
                    if (!whole && (add == out || b0 > 0)) add = nullptr;        // what is in `out` already, or the first share's to bring
#pragma unroll
                    for (int j = 0; j < TPW; j++) {
                        const long long tok = (long long)tt * NT + cg * TPW + j;
                        if (tok >= a.T) continue;
                        const unsigned long long v = sum[j] + (add ? (unsigned long long)add[tok * out_f + row] : 0ULL);
                        if (whole) out[tok * out_f + row] = (int64_t)v;
                        else atomicAdd(reinterpret_cast<unsigned long long *>(out + tok * out_f + row), v);      // exact in any order
                    }
                }
#pragma unroll
                for (int j = 0; j < TPW; j++) sum[j] = 0;
            }
        };
        if (np == 3) read_out(std::integral_constant<int, 3>{});
        else if (np == 4) read_out(std::integral_constant<int, 4>{});
        else if (np == 6) read_out(std::integral_constant<int, 6>{});
        else read_out(std::integral_constant<int, 8>{});
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp < QC_MMA_WARP) {
        // ================= expansion: bits -> bytes +1 / -1, two 16-row sub-tiles per warp ======================
        const int ew = warp - QC_READ, g = lane >> 2, t = lane & 3;
        // MMA m of a block covers columns 32 m .. 32 m + 31; this lane's eight bytes of it are half of 16-byte chunk
        // 2 m + (t >> 1) of its row.  Lanes of odd g take their two words in the other order, so that the 16 lanes of a store
        // phase fall on all banks of the swizzled row group.
        uint32_t off[4];
#pragma unroll
        for (int m = 0; m < 4; m++) off[m] = (uint32_t)(ew * 32 * 128 + g * 128 + (((2 * (m ^ (2 * (g & 1))) + (t >> 1)) ^ g) << 4) + (t & 1) * 8);
        Ring unit, st;
        bool ok = true;
        for (long long u = u0; u < u1 && ok;) {
            const int b0 = (int)(u % nb), b1 = (int)min((long long)nb, b0 + (u1 - u));
            u += b1 - b0;
            for (int b = b0; b < b1; b++) {
                if (b == b0 || (b & (QC_CHUNK - 1)) == 0) {
                    ok = qc_wait_warp(raw_full + 8 * unit.slot, unit.pass, &s_abort);
                    if (!ok) break;
                }
                const unsigned char *bits = raw + unit.slot * RAW_BYTES + (b & (QC_CHUNK - 1)) * US + ew * 2 * (QC_CHUNK * US) + lane * 8;
                uint2 w[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(bits + h * (QC_CHUNK * US));
                    w[h] = (g & 1) ? make_uint2(v.y, v.x) : v;
                }
                if (st.lapped) {
                    ok = qc_wait_warp(empty_bar + 8 * st.slot, st.pass ^ 1, &s_abort);
                    if (!ok) break;
                }
                const uint32_t dst = qc_u32(smem + st.slot * stage_bytes);
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int m = 0; m < 4; m++)
#pragma unroll
                        for (int hi = 0; hi < 2; hi++) {           // rows g and g + 8; byte columns 0..3 and 4..7
                            const uint32_t word = m >> 1 ? w[h].y : w[h].x;
                            const int r0 = 4 * (m & 1) + hi;
                            // bit 1 -> 0x01, bit 0 -> 0xFF: 0xFF - 0xFE * bit in every byte
                            const uint32_t x0 = ((word >> r0) & 0x01010101u) * 0xFFFFFF02u + 0xFFFFFFFFu;
                            const uint32_t x1 = ((word >> (r0 + 2)) & 0x01010101u) * 0xFFFFFF02u + 0xFFFFFFFFu;
                            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + off[m] + h * 2048 + hi * 1024), "r"(x0), "r"(x1) : "memory");
                        }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) qc_arrive(full_bar + 8 * st.slot);
                st.step(stages);
                if (b + 1 == b1 || ((b + 1) & (QC_CHUNK - 1)) == 0) unit.step(QC_RAW_SLOTS);
            }
        }
    } else if (warp == QC_MMA_WARP) {
        // ================= MMAs ===============================================================================
        // (the whole warp walks the loop, so that its addresses stay in uniform registers; one elected lane issues)
        const bool two = cols > 256;                               // more columns than one instruction takes: two halves
        const int n_mma = two ? cols / 2 : cols;
        const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n_mma >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);     // s8 x s8 -> s32
        const uint32_t leader = qc_elect();
        const int n = (int)(u1 - u0);
        Ring st, buf;
        for (int i = 0; i < n; i++) {
            if (!qc_wait_warp(full_bar + 8 * st.slot, st.pass, &s_abort)) break;
            if (buf.lapped && !qc_wait_warp(free_bar + 8 * buf.slot, buf.pass ^ 1, &s_abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t stage = qc_u32(smem + st.slot * stage_bytes), d = tmem + buf.slot * buf_cols;
            const uint64_t da = qc_desc(stage), db = qc_desc(stage + QC_A_BYTES);
            if (leader) {
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    qc_mma(d, da + ks * 2, db + ks * 2, idesc, ks);
                    if (two) qc_mma(d + n_mma, da + ks * 2, db + n_mma * 8 + ks * 2, idesc, ks);
                }
                qc_commit(empty_bar + 8 * st.slot);
                qc_commit(acc_bar + 8 * buf.slot);
            }
            __syncwarp();
            st.step(stages); buf.step(nbuf);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp == QC_PLANE_WARP) {
        // ================= digit planes of the tile's tokens ==================================================
        if (lane == 0) {
            Ring st;
            bool ok = true;
            for (long long u = u0; u < u1 && ok;) {
                const long long tl = u / nb;
                const int b0 = (int)(u - tl * nb), b1 = (int)min((long long)nb, b0 + (u1 - u));
                int p, rt, tt;
                locate(t0 + tl * tstep, p, rt, tt);
                u += b1 - b0;
                for (int b = b0; b < b1; b++) {
                    if (st.lapped && !(ok = qc_wait(empty_bar + 8 * st.slot, st.pass ^ 1, &s_abort))) break;
                    const uint32_t dst = qc_u32(smem + st.slot * stage_bytes + QC_A_BYTES);
                    qc_expect(full_bar + 8 * st.slot, cols * 128);
                    for (int l = 0; l < mp; l++)
                        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                                     ::"r"(dst + l * NT * 128), "l"(reinterpret_cast<uint64_t>(&xmap)), "r"(b * 128), "r"(l), "r"(tt * NT),
                                       "r"(full_bar + 8 * st.slot) : "memory");
                    st.step(stages);
                }
            }
            // given up: the copies in flight land before the CTA leaves (a slot behind the ring's position is in its previous lap)
            if (!ok) for (int s = 0; s < stages; s++)
                for (unsigned it = 0; it < QC_WAIT_LIMIT && !qc_try(full_bar + 8 * s, s < st.slot ? st.pass : st.pass ^ 1); it++) {}
        }
    } else {
        // ================= registered units: eight blocks of the eight sub-tiles per slot ======================
        Ring unit;
        bool ok = true;
        for (long long u = u0; u < u1 && ok;) {
            const long long tl = u / nb;
            const int b0 = (int)(u - tl * nb), b1 = (int)min((long long)nb, b0 + (u1 - u));
            int p, rt, tt;
            locate(t0 + tl * tstep, p, rt, tt);
            const long long tile16 = (long long)rt * 8 + lane, n16 = (a.part[p].out_f + 15) / 16;
            const int live = (int)min(8LL, n16 - (long long)rt * 8);             // sub-tiles the matrix has
            u += b1 - b0;
            for (int b = b0; b < b1;) {
                const int n = min(QC_CHUNK - (b & (QC_CHUNK - 1)), b1 - b);
                const int slot = unit.slot;
                if (unit.lapped && !(ok = qc_wait_warp(raw_empty + 8 * slot, unit.pass ^ 1, &s_abort))) break;
                if (lane == 0) qc_expect(raw_full + 8 * slot, live * n * US);
                __syncwarp();
                if (lane < live)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(qc_u32(raw + slot * RAW_BYTES + lane * (QC_CHUNK * US) + (b & (QC_CHUNK - 1)) * US)),
                                   "l"(a.part[p].units + (tile16 * nb + b) * US), "r"(n * US), "r"(raw_full + 8 * slot) : "memory");
                unit.step(QC_RAW_SLOTS);
                b += n;
            }
        }
        if (!ok && lane == 0) for (int c = 0; c < QC_RAW_SLOTS; c++)
            for (unsigned it = 0; it < QC_WAIT_LIMIT && !qc_try(raw_full + 8 * c, c < unit.slot ? unit.pass : unit.pass ^ 1); it++) {}
    }
    __syncthreads();
    if (warp == QC_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (tid == 0 && s_abort && a.flags) atomicOr(a.flags, 8);
}

using QcEncode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
QcEncode qc_encode() {
    static QcEncode fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<QcEncode>(p);
    }();
    return fn;
}

// token tile: the read-out and the planes grow with it, the expansion of the signs does not
int qc_tile_tokens(long long T) { return T <= 8 ? 8 : T <= 16 ? 16 : T <= 32 ? 32 : 64; }

template <int NT, typename DT>
cudaError_t launch_tc(Q1TcArgs a, const int8_t *planes, cudaStream_t s) {
    QcEncode enc = qc_encode();
    if (!enc) return cudaErrorNotSupported;
    const long long K = (long long)a.nb * 128;
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)K, 8, (cuuint64_t)a.T};
    const cuuint64_t strides[2] = {(cuuint64_t)K, (cuuint64_t)(8 * K)};
    const cuuint32_t box[3] = {128, 1, NT}, estr[3] = {1, 1, 1};
    if (enc(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t *>(planes), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(q1_tc_kernel<NT, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, QC_SMEM);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    a.n_ttiles = (int)((a.T + NT - 1) / NT);
    a.n_tiles = (long long)a.tile_end[a.n_parts - 1] * a.n_ttiles;
    // four whole tiles per SM keep the last wave's loss below the cost of the partial sums; below that the blocks are dealt
    // out, at least four to a CTA (less would be all start-up)
    a.split = q1_tc_split(a.tile_end[a.n_parts - 1], a.T);
    long long grid = std::min<long long>(Q1_TC_CTAS, a.n_tiles);
    if (a.split) grid = std::min<long long>(Q1_TC_CTAS, std::max<long long>(1, a.n_tiles * a.nb / 4));
    launch_behind(q1_tc_kernel<NT, DT>, (unsigned)grid, qc_threads(NT), QC_SMEM, s, a, map);
    note_launch();
    return cudaGetLastError();
}

}  // namespace

bool q1_tc_split(long long row_tiles, long long T) {
    const int nt = qc_tile_tokens(T);
    return row_tiles * ((T + nt - 1) / nt) < 4 * Q1_TC_CTAS;
}

cudaError_t launch_q1_tc(const Q1Part *parts, int n_parts, bool sc32, long long nb, const int8_t *planes, long long T, int sh,
                         const int *nl_dev, cudaStream_t s) {
    if (n_parts < 1 || n_parts > Q1_MAX_PARTS || nb <= 0 || nb > (1 << 20) || T <= 0 || !nl_dev || (reinterpret_cast<uintptr_t>(planes) & 15)) return cudaErrorInvalidValue;
    Q1TcArgs a = {};
    a.n_parts = n_parts; a.nb = (int)nb; a.T = T; a.sh = sh; a.nl_dev = nl_dev; a.flags = shared_flag_word();
    unsigned long long max_scale = 0;
    for (int p = 0; p < n_parts; p++) {
        max_scale = std::max(max_scale, parts[p].max_scale);
        a.part[p] = parts[p];
        a.tile_end[p] = (p ? a.tile_end[p - 1] : 0) + (int)((parts[p].out_f + 127) / 128);
    }
    // three digit planes: |sum over a block| <= 128 * 8421504 (all digits -128), so that the products of a tile, taken down to the shift
    // (less than 2^32 a block), add up to less than 1077952512 * (2^33 - 2^26) + 2^52 < 2^63
    a.narrow = sh < 32 && max_scale < (1ULL << 32) && max_scale * (unsigned long long)nb < (1ULL << 33) - (1ULL << 26);
    const int nt = qc_tile_tokens(T);
    if (nt == 8) return sc32 ? launch_tc<8, int>(a, planes, s) : launch_tc<8, long long>(a, planes, s);
    if (nt == 16) return sc32 ? launch_tc<16, int>(a, planes, s) : launch_tc<16, long long>(a, planes, s);
    if (nt == 32) return sc32 ? launch_tc<32, int>(a, planes, s) : launch_tc<32, long long>(a, planes, s);
    return sc32 ? launch_tc<64, int>(a, planes, s) : launch_tc<64, long long>(a, planes, s);
}

}  // namespace iie
