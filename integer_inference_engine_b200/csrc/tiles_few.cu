// Gate / up products of experts with few rows each (Q4_K) on the tcgen05 tiles: tiles of eight rows, unscaled weight codes.
//
// What bounds the tiles of tiles.cu at few rows is the expansion of a weight to two bytes: a multiplication and two stores per four
// weights and byte plane, whatever the rows (6750 warp instructions per 128 x 256 weights).  Here the A operand is the packed code itself, one byte with the other nibble masked
// (q, or 16 q), and every sub-block of 32 columns, one MMA step, has accumulators of its own:
//     D_j = sum over the sub-block of q x_l,  j = 0..7,  for eight rows x four digits l (MMA N = 32),
// so that the sub-block scales are applied at the read-out, T_l = sum_j sc_j D_j (32 bits, once per sub-block, row and digit), the
// block scale d and the minima as in tiles.cu.  That moves the work from the weights to the rows: two instructions a word of codes, and
// 24 multiply-adds per column and weight row of a super-block.  4800 warp instructions per 128 x 256 weights, 2200 clocks: the read-out of a
// super-block is a chain of waits and loads, with six warps a scheduler at 0.57 instructions per clock.  Gate / up of 128 experts of 768 x
// 2048, 64 tokens: 135 -> 114 us (HBM 33).  Two teams of read-out warps that take turns: 135; both warps of a row on the same four columns
// where a tile has no more: 115; the planes by TMA boxes of one plane instead of four: 113.
// Activations of more than four digits walk the super-blocks twice, digits 0..3 and 4..7.
//
// Roles (23 warps): eight read-out warps (lane = weight row, four columns each; a half tile without live columns is not read), eight
// expanding warps (two half-tiles each, a whole super-block per stage), MMAs, TMA loads of planes and sums, bulk copies of weights,
// four epilogue warps (SiLU * up, digit planes).  Accumulators: three buffers of half a super-block (4 x 32 columns) and two of the
// minima's products (six digits of the sums x eight rows).  Every wait is bounded, see tiles.cu.
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "layout.cuh"
#include "mma_items.cuh"
#include "tile_ops.cuh"

namespace iie {

namespace {

constexpr int TF_BN = 8, TF_READ = 8, TF_EXPAND = 8, TF_EPI = 4;
constexpr int TF_MMA_WARP = TF_READ + TF_EXPAND, TF_X_WARP = TF_MMA_WARP + 1, TF_W_WARP = TF_MMA_WARP + 2, TF_EPI_WARP = TF_MMA_WARP + 3;
constexpr int TF_THREADS = (TF_EPI_WARP + TF_EPI) * 32;
constexpr int TF_PANEL = 128 * 128;                                // 128 weight rows x half a super-block of codes
constexpr int TF_MINS = 128 * 32, TF_PLANES = 4, TF_X_PANEL = TF_PLANES * TF_BN * 128, TF_SUMS = 6, TF_S_BYTES = TF_SUMS * TF_BN * 32;
constexpr int TF_X = 2 * TF_PANEL, TF_M = TF_X + 2 * TF_X_PANEL, TF_S = TF_M + TF_MINS;        // offsets in a stage
constexpr int TF_STAGE = (TF_S + TF_S_BYTES + 1023) & ~1023, TF_STAGES = 3;
constexpr int TF_RAW_BYTES = 16 * HTB_Q4K, TF_RAW = 3;
constexpr int TF_EXCH = TF_BN * 128 * 8;
constexpr int TF_SMEM = 1024 + TF_STAGES * TF_STAGE + TF_EXCH + TF_RAW * TF_RAW_BYTES;
constexpr int TF_HALVES = 3, TF_HALF_COLS = 4 * 32, TF_MIN_COL = TF_HALVES * TF_HALF_COLS, TF_MIN_COLS = TF_SUMS * TF_BN;
constexpr int TF_MAX_GROUPS = 1024;
static_assert(TF_SMEM <= 217 * 1024 && TF_MIN_COL + 2 * TF_MIN_COLS <= 512, "");

__device__ __forceinline__ void tl_ld16(uint32_t addr, int (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(addr));
}
__device__ __forceinline__ void tl_ld_sums(uint32_t addr, int (&r)[4]) { tl_ld4(addr, r); }
__device__ __forceinline__ void tl_ld_sums(uint32_t addr, int (&r)[6]) {
    int q[4];
    tl_ld4(addr, q);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[4]), "=r"(r[5]) : "r"(addr + 4));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    r[0] = q[0]; r[1] = q[1]; r[2] = q[2]; r[3] = q[3];
}
struct FewMaps { CUtensorMap x, s; };                              // four planes and six digits of the sums, of eight rows each: N = row x digit

__global__ void __launch_bounds__(TF_THREADS, 1) tile_few_kernel(const TileArgs a, const __grid_constant__ FewMaps maps) {
    extern __shared__ __align__(1024) unsigned char tf_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tf_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *exch = smem + TF_STAGES * TF_STAGE, *raw = exch + TF_EXCH;
    __shared__ __align__(8) uint64_t bars[2 * TF_STAGES + 2 * TF_HALVES + 2 * TF_RAW + 2];
    __shared__ int s_first[TF_MAX_GROUPS + 1], s_off[TF_MAX_GROUPS + 1];       // first tile and first row of each group
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const uint32_t full_bar = tl_u32(bars), empty_bar = full_bar + 8 * TF_STAGES, acc_bar = empty_bar + 8 * TF_STAGES, free_bar = acc_bar + 8 * TF_HALVES,
                   raw_full = free_bar + 8 * TF_HALVES, raw_empty = raw_full + 8 * TF_RAW, y_full = raw_empty + 8 * TF_RAW, y_free = y_full + 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nb = a.nb;
    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < TF_STAGES; s++) { tl_init(full_bar + 8 * s, TF_EXPAND + 1); tl_init(empty_bar + 8 * s, 1); }
        for (int s = 0; s < TF_HALVES; s++) { tl_init(acc_bar + 8 * s, 1); tl_init(free_bar + 8 * s, TF_READ); }
        for (int s = 0; s < TF_RAW; s++) { tl_init(raw_full + 8 * s, 1); tl_init(raw_empty + 8 * s, TF_READ + TF_EXPAND); }
        tl_init(y_full, TF_READ); tl_init(y_free, TF_EPI);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TF_X_WARP && lane == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.x)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.s)) : "memory");
    }
    if (a.few == 2) {                                              // the kernel before knows which form takes the call
        pdl_enter();
        if (*a.form) return;
    }
    if (warp == TF_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tl_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (a.few != 2) pdl_enter();                                   // what stands above needs nothing of the kernel before
    const int np = tl_planes(a.x_nl ? max(1, min(8, *a.x_nl)) : 8), walks = np > TF_PLANES ? 2 : 1;       // uniform over the grid
    const int n_rt = (int)((a.out_f + 63) / 64);
    if (tid == 0 && blockIdx.x == 0) { atomicAdd(a.counts + (np == 3 ? 0 : np == 4 ? 1 : 7), 1ULL); atomicAdd(a.counts + TILE_SHAPES + 2, 1ULL); }      // (as a gate / up tile of tiles.cu, too)
    if (warp == 0) {                                               // first tile of every group
        int base = 0;
        for (int g0 = 0; g0 < a.n_groups; g0 += 32) {
            const int g = g0 + lane;
            const int at = g < a.n_groups ? a.grp_off[g] : 0, rows = g < a.n_groups ? a.grp_off[g + 1] - at : 0;
            const int nt = (rows + TF_BN - 1) / TF_BN * n_rt;
            int incl = nt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, d); if (lane >= d) incl += t; }
            if (g < a.n_groups) { s_first[g] = base + incl - nt; s_off[g] = at; if (g + 1 == a.n_groups) s_off[g + 1] = at + rows; }
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_first[a.n_groups] = base;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const int n_tiles = s_first[a.n_groups];

    // tile -> group, row tile, first and past-the-last activation row
    struct Where { int g, rt, m0, m_end; };
    auto locate = [&](int tile) {
        int lo = 0, hi = a.n_groups;                               // s_first[lo] <= tile < s_first[hi]
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_first[mid] <= tile) lo = mid; else hi = mid; }
        const int first = s_off[lo], end = s_off[lo + 1], nt = (end - first + TF_BN - 1) / TF_BN, i = tile - s_first[lo];
        Where w;
        w.g = lo; w.rt = i / nt; w.m0 = first + (i - w.rt * nt) * TF_BN; w.m_end = end;
        return w;
    };
    const int n_ht = (int)((a.out_f + 7) >> 3);

    if (warp < TF_READ) {
        // ================= read-out ===========================================================================
        const int rowt = (warp & 3) * 32 + lane, cg = warp >> 2;
        const uint32_t quarter = tmem + ((uint32_t)((warp & 3) * 32) << 16), tlane = quarter + cg * 16, tmin = quarter + TF_MIN_COL + cg * 4 * TF_SUMS;
        const int meta_off = (rowt >> 3) * HTB_Q4K + 1024 + (rowt & 7) * 16;
        // SHORT: up to three digits, so that two 64-bit sums 16 bits apart and four digits of the sub-block sums do
        auto read_out = [&](auto short_c) {
            constexpr bool SHORT = decltype(short_c)::value;
            constexpr int ND = SHORT ? 3 : 4, NLV = SHORT ? 2 : 5;
            TlRing rs, buf;
            int min_slot = 0;
            uint32_t y_pass = 0;
            bool y_used = false, ok = true;
            for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
                const Where w = locate(tile);
                const bool live = w.m0 + cg * 4 < w.m_end;         // columns of this warp with rows behind them
                long long L[NLV][4];
#pragma unroll
                for (int i = 0; i < NLV; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) L[i][j] = 0;
#pragma unroll
                for (int walk = 0; walk < (SHORT ? 1 : 2); walk++) {
                    if (walk >= walks) break;
                    for (int b = 0; b < nb; b++) {
                        if (!(ok = tl_wait(raw_full + 8 * rs.slot, rs.pass, &s_abort))) break;
                        const uint4 meta = *reinterpret_cast<const uint4 *>(raw + rs.slot * TF_RAW_BYTES + meta_off);
                        __syncwarp();
                        if (lane == 0) tl_arrive(raw_empty + 8 * rs.slot);
                        rs.step(TF_RAW);
                        const int d = scale_small(meta.x & 0xFFFF, a.fw), dm = -scale_small(meta.x >> 16, a.fw), d8 = d << 8;
                        uint32_t sc[2], mn[2];
                        q4k_scales(meta.y, meta.z, meta.w, sc[0], sc[1], mn[0], mn[1]);
                        int T[ND][4];
#pragma unroll
                        for (int l = 0; l < ND; l++)
#pragma unroll
                            for (int j = 0; j < 4; j++) T[l][j] = 0;
#pragma unroll
                        for (int half = 0; half < 2; half++) {
                            if (!(ok = tl_wait(acc_bar + 8 * buf.slot, buf.pass, &s_abort))) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            if (live) {
                                const uint32_t base = tlane + buf.slot * TF_HALF_COLS;
#pragma unroll
                                for (int q = 0; q < 4; q += 2) {   // sub-blocks 4 half + q (low nibbles), q + 1 (high nibbles, 16 times the codes)
                                    int r[2][16];                  // four rows x four digits
#pragma unroll
                                    for (int u = 0; u < 2; u++) tl_ld16(base + (q + u) * 32, r[u]);
                                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                                    const int s0 = ubyte_at(sc[half], q) * 16, s1 = ubyte_at(sc[half], q + 1);
#pragma unroll
                                    for (int l = 0; l < ND; l++)
#pragma unroll
                                        for (int j = 0; j < 4; j++) T[l][j] += r[0][4 * j + l] * s0 + r[1][4 * j + l] * s1;      // 16 T, below 2^29
                                }
                                if (half == 0) {                   // the minima's product: digits 0..5 of the sums, behind the first walk 6..8
                                    constexpr int NS = SHORT ? 4 : 6;
                                    int r[4][NS];
#pragma unroll
                                    for (int j = 0; j < 4; j++) tl_ld_sums(tmin + min_slot * TF_MIN_COLS + j * TF_SUMS, r[j]);
                                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                                    for (int l = 0; l < NS; l += 2)
#pragma unroll
                                        for (int j = 0; j < 4; j++) {
                                            const int i = (walk ? 3 : 0) + l / 2;
                                            if (i < NLV) L[i < NLV ? i : 0][j] += (long long)(r[j][l] + r[j][l + 1] * 256) * (long long)dm;
                                        }
                                }
                            }
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) tl_arrive(free_bar + 8 * buf.slot);
                            buf.step(TF_HALVES);
                        }
                        if (!ok) break;
                        min_slot ^= 1;
                        if (live) {
#pragma unroll
                            for (int l = 0; l < ND; l++) {
                                if (!SHORT && 4 * walk + l >= np) break;           // (digits that are not in use stand for nothing)
#pragma unroll
                                for (int j = 0; j < 4; j++) L[2 * walk + l / 2][j] += (long long)(T[l][j] >> 4) * (long long)((l & 1) ? d8 : d);
                            }
                        }
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                // ---- y = floor(V / 2^fw) to the epilogue warps ------------------------------------------------
                if (y_used && !(ok = tl_wait(y_free, y_pass ^ 1, &s_abort))) break;
                long long *to = reinterpret_cast<long long *>(exch) + cg * 4 * 128 + rowt;
                if (live) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        i128 v = L[NLV - 1][j];
#pragma unroll
                        for (int i = NLV - 2; i >= 0; i--) v = (v << 16) + (i128)L[i][j];
                        to[j * 128] = (long long)(v >> a.fw);
                    }
                }
                __syncwarp();
                if (lane == 0) tl_arrive(y_full);
                y_used = true; y_pass ^= 1;
            }
        };
        if (np <= 3) read_out(std::true_type{}); else read_out(std::false_type{});
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp < TF_MMA_WARP) {
        // ================= expansion: packed codes -> bytes, a super-block per stage =============================
        const int ew = warp - TF_READ, g = lane >> 2, t = lane & 3;
        // sub-block m of a half: this lane's eight bytes are half of 16-byte chunk 2 m + (t >> 1) of its row; lanes of odd g take their two
        // groups in the other order, so that the 16 lanes of a store phase fall on all banks
        uint32_t off[4];
#pragma unroll
        for (int i = 0; i < 4; i++) off[i] = (uint32_t)(g * 128) + ((((2 * (i ^ (2 * (g & 1))) + (t >> 1)) ^ g) << 4) + (t & 1) * 8);
        TlRing rs, st;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x)
            for (int i = 0, b = 0; i < walks * nb; i++, b = b + 1 == nb ? 0 : b + 1) {
                if (!(ok = tl_wait(raw_full + 8 * rs.slot, rs.pass, &s_abort))) break;
                const unsigned char *slot = raw + rs.slot * TF_RAW_BYTES;
                uint4 q_in[2][2], meta[2];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned char *unit = slot + (ew + TF_EXPAND * h) * HTB_Q4K;
                    q_in[h][0] = *reinterpret_cast<const uint4 *>(unit + lane * 16); q_in[h][1] = *reinterpret_cast<const uint4 *>(unit + 512 + lane * 16);
                    meta[h] = *reinterpret_cast<const uint4 *>(unit + 1024 + g * 16);
                }
                __syncwarp();
                if (lane == 0) tl_arrive(raw_empty + 8 * rs.slot);
                rs.step(TF_RAW);
                if (st.lapped && !(ok = tl_wait(empty_bar + 8 * st.slot, st.pass ^ 1, &s_abort))) break;
                const uint32_t dst = tl_u32(smem + st.slot * TF_STAGE);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int unit = ew + TF_EXPAND * h;
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        uint4 q = q_in[h][p];
                        if (g & 1) q = make_uint4(q.z, q.w, q.x, q.y);
                        const uint32_t to = dst + p * TF_PANEL + unit * 1024;      // eight rows of 128 bytes
                        tl_sts64(to + off[0], q.x & 0x0f0f0f0fu, q.y & 0x0f0f0f0fu);
                        tl_sts64(to + off[1], q.x & 0xf0f0f0f0u, q.y & 0xf0f0f0f0u);
                        tl_sts64(to + off[2], q.z & 0x0f0f0f0fu, q.w & 0x0f0f0f0fu);
                        tl_sts64(to + off[3], q.z & 0xf0f0f0f0u, q.w & 0xf0f0f0f0u);
                    }
                    uint32_t sc[2], mn[2];                         // the row's eight minima, in the columns of this super-block's sums
                    q4k_scales(meta[h].y, meta[h].z, meta[h].w, sc[0], sc[1], mn[0], mn[1]);
                    const int r = unit * 8 + g;
                    const bool mine = t == (b & 3);
                    tl_sts64(dst + TF_M + r * 32 + (((t >> 1) ^ ((r >> 2) & 1)) << 4) + (t & 1) * 8, mine ? mn[0] : 0, mine ? mn[1] : 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tl_arrive(full_bar + 8 * st.slot);
                st.step(TF_STAGES);
            }
    } else if (warp == TF_MMA_WARP) {
        // ================= MMAs (the whole warp walks the loop, one elected lane issues) ===============================
        const uint32_t leader = tl_elect();
        const uint32_t id_x = tl_idesc(TF_PLANES * TF_BN, false), id_min = tl_idesc(TF_MIN_COLS, false);
        TlRing st, buf;
        int min_slot = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x)
            for (int i = 0; i < walks * nb && ok; i++) {
                if (!(ok = tl_wait(full_bar + 8 * st.slot, st.pass, &s_abort))) break;
                const uint32_t stage = tl_u32(smem + st.slot * TF_STAGE);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    if (buf.lapped && !(ok = tl_wait(free_bar + 8 * buf.slot, buf.pass ^ 1, &s_abort))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + buf.slot * TF_HALF_COLS;
                    const uint64_t da = tl_desc128(stage + half * TF_PANEL), db = tl_desc128(stage + TF_X + half * TF_X_PANEL);
                    if (leader) {
#pragma unroll
                        for (int j = 0; j < 4; j++) tl_mma(d + j * 32, da + j * 2, db + j * 2, id_x, 0);
                        if (half == 0) tl_mma(tmem + TF_MIN_COL + min_slot * TF_MIN_COLS, tl_desc32(stage + TF_M), tl_desc32(stage + TF_S), id_min, 0);
                        if (half == 1) tl_commit(empty_bar + 8 * st.slot);
                        tl_commit(acc_bar + 8 * buf.slot);
                    }
                    __syncwarp();
                    buf.step(TF_HALVES);
                }
                st.step(TF_STAGES); min_slot ^= 1;
            }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp == TF_X_WARP) {
        // ================= digit planes and sub-block sums of the tile's rows ==================================
        if (lane == 0) {
            TlRing st;
            bool ok = true;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                const Where w = locate(tile);
                for (int i = 0, b = 0, walk = 0; i < walks * nb; i++) {
                    const uint32_t eb = empty_bar + 8 * st.slot, fb = full_bar + 8 * st.slot;
                    if (st.lapped && !(ok = tl_try(eb, st.pass ^ 1) || tl_wait_slow(eb, st.pass ^ 1, &s_abort))) break;
                    const uint32_t dst = tl_u32(smem + st.slot * TF_STAGE);
                    tl_expect(fb, 2 * TF_X_PANEL + TF_S_BYTES);
                    for (int half = 0; half < 2; half++) tl_tma(dst + TF_X + half * TF_X_PANEL, &maps.x, b * 256 + half * 128, walk * TF_PLANES, w.m0, fb);
                    tl_tma(dst + TF_S, &maps.s, (b >> 2) * 32, walk * TF_SUMS, w.m0, fb);      // (digits beyond nine: zeros)
                    st.step(TF_STAGES);
                    if (++b == nb) { b = 0; walk++; }
                }
            }
            // given up: the copies in flight land before the CTA leaves (a slot behind the ring's position is in its current lap)
            if (!ok) for (int s = 0; s < TF_STAGES; s++)
                for (unsigned it = 0; it < TL_WAIT_LIMIT && !tl_try(full_bar + 8 * s, s < st.slot ? st.pass : st.pass ^ 1); it++) {}
        }
    } else if (warp == TF_W_WARP) {
        // ================= packed weights: one super-block of the tile's 16 half-tiles per slot ===============
        TlRing rs;
        bool ok = true;
        for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const Where w = locate(tile);
            const int ht = w.rt * 8 + (lane & 7);
            const bool live = lane < 16 && ht < n_ht;
            const uint8_t *src = live ? (lane >= 8 ? a.wb[w.g] : a.wa[w.g]) + (long long)ht * nb * HTB_Q4K : nullptr;
            const int n_live = __popc(__ballot_sync(0xffffffffu, live));
            for (int i = 0, b = 0; i < walks * nb; i++, b = b + 1 == nb ? 0 : b + 1) {
                const uint32_t eb = raw_empty + 8 * rs.slot, fb = raw_full + 8 * rs.slot;
                if (rs.lapped && !(ok = tl_wait(eb, rs.pass ^ 1, &s_abort))) break;
                if (lane == 0) tl_expect(fb, n_live * HTB_Q4K);
                __syncwarp();
                if (live) asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                       ::"r"(tl_u32(raw + rs.slot * TF_RAW_BYTES + lane * HTB_Q4K)), "l"(src + (long long)b * HTB_Q4K), "r"(HTB_Q4K), "r"(fb) : "memory");
                rs.step(TF_RAW);
            }
        }
        if (!ok && lane == 0) for (int s = 0; s < TF_RAW; s++)
            for (unsigned it = 0; it < TL_WAIT_LIMIT && !tl_try(raw_full + 8 * s, s < rs.slot ? rs.pass : rs.pass ^ 1); it++) {}
    } else {
        // ================= SiLU(g) * u and its digit planes ====================================================
        const int et = tid - TF_EPI_WARP * 32, r = et & 63, part = et >> 6;      // output row of the tile, odd or even columns
        int nl_max = 0;
        uint32_t pass = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const Where w = locate(tile);
            const long long row = (long long)w.rt * 64 + r;
            if (!tl_wait(y_full, pass, &s_abort)) break;
            const int n = min(TF_BN, w.m_end - w.m0);
            const long long *from = reinterpret_cast<const long long *>(exch) + part * 128 + r;
            int64_t gu[TF_BN / 2];
            bool least = false;
#pragma unroll
            for (int i = 0; i < TF_BN / 2; i++) {
                gu[i] = 0;
                if ((i & ~1) * 2 < n) {                            // four columns at a time
                    const int64_t g = from[2 * i * 128];
                    least |= g == INT64_MIN;
                    gu[i] = silu_up_fixed(g, from[2 * i * 128 + 64], a.fa, a.sig_log2e, a.sig_clip);
                }
            }
            if (least)
#pragma unroll
                for (int i = 0; i < TF_BN / 2; i++) gu[i] = silu_up_any(from[2 * i * 128], from[2 * i * 128 + 64], a.fa, a.sig_log2e, a.sig_clip);
            __syncwarp();
            if (lane == 0) tl_arrive(y_free);
            pass ^= 1;
#pragma unroll
            for (int i = 0; i < TF_BN / 2; i++) {
                const int c = 2 * i + part, col = w.m0 + c;
                if (c >= n || row >= a.out_f) continue;
                bool fits;
                const uint64_t dg = balanced_digits8(gu[i], fits);
                if (!fits) atomicOr(a.flags, 1);
                nl_max = max(nl_max, digits_used(dg));
                if (a.out) a.out[(long long)col * a.out_f + row] = gu[i];
                int8_t *ol = a.out_limbs + (long long)col * 8 * a.out_f + row;
#pragma unroll
                for (int l = 0; l < 8; l++) ol[l * a.out_f] = (int8_t)(dg >> (8 * l));
            }
        }
        if (a.out_nl) {
            nl_max = __reduce_max_sync(0xffffffffu, nl_max);
            if (lane == 0 && nl_max > 0) atomicMax(a.out_nl, nl_max);
        }
    }
    __syncthreads();
    if (warp == TF_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (tid == 0 && s_abort) atomicOr(a.flags, 8);
}

}  // namespace

// x: digit planes in pair order (or row order without `xidx`); a.xs filled.  The caller has checked shapes and scales (launch_tiles).
cudaError_t launch_tiles_few(const TileArgs &a, const int8_t *x, cudaStream_t s) {
    FewMaps maps;
    const long long K = (long long)a.nb * 256;
    const int stride = (a.nb * 8 + 31) / 32 * 32;
    if (!tl_map(&maps.x, x, K, 8, a.n_rows, 128, TF_BN, CU_TENSOR_MAP_SWIZZLE_128B, TF_PLANES) ||
        !tl_map(&maps.s, a.xs, stride, 9, a.n_rows, 32, TF_BN, CU_TENSOR_MAP_SWIZZLE_32B, TF_SUMS))
        return cudaErrorInvalidValue;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(tile_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TF_SMEM);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    const long long most = (a.n_rows / TF_BN + std::min<long long>(a.n_groups, a.n_rows)) * ((a.out_f + 63) / 64);
    launch_behind(tile_few_kernel, (unsigned)std::max<long long>(1, std::min<long long>(148, most)), TF_THREADS, TF_SMEM, s, a, maps);
    note_launch();
    return cudaGetLastError();
}

}  // namespace iie
