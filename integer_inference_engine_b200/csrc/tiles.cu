// Grouped and dense fused-dequant products of two rows and more on the 5th-generation tensor cores (tcgen05, kind::i8).
//
// Replaces the reference's pair-parallel prefill kernels (north-mini-code/tools/nmc_qk_cuda.cu:2184-2201 matmul_multi_tok /
// combine_tok and the host loop :2203-2346), which stream one expert's weights once per (token, expert) pair.
//
// y = floor(V / 2^fw), V = sum over the 256-column super-blocks of  d * T - dmin * M  with
//     T = sum_k (sc_k q_k) x_k            (Q4_K: sc < 64, q < 16; Q6_K: sc int8, q - 32 in its place, dmin = 0)
//     M = sum_j m_j S_j,  S_j = sum of the 32 x of sub-block j.
// The tensor cores form T and M of ONE super-block, the block scales are applied when its accumulators are read out.  That
// keeps the weight operand at two bytes: sc q (Q4_K, times 16, below 2^14) and sc (q - 32) (Q6_K, |.| <= 4096) are 16-bit
// numbers, low byte unsigned, high byte unsigned / signed.  Where the instructions of the expansion bound the tile (Q4_K, sixteen
// columns), the bytes are sl q and sh q with sc = 8 sh + sl: four of them per multiplication, for np - 1 accumulators more.  (Dequantising fully, W = d sc q - dmin m, takes four or five signed
// digits: twice the multiplications and four times the instructions to expand a weight.)  With x in np digits x_l and S in
// ns = np + 1:  T = sum_{a,l} 256^(a+l) A_a x_l is 2 np products into np + 1 accumulators, M one product of a 32-column step
// (eight m per super-block) with the sums' digits.  Everything stays exact: |acc_s| < 2^25, and in the read-out
// V = sum_i 2^(16 i) L_i with L_i += acc_2i * d + acc_2i+1 * 256 d - ... in 64 bits, put together in 128 bits once per tile.
//
// Tile: 128 weight rows (MMA M, TMEM lanes) x bn rows of the activation (bn = 16 or 32); the digit planes of the rows are stacked
// along N, so a K step is two MMAs (one per weight byte) whatever np is.  Gate and up rows share a tile (lanes 0..63 gate, 64..127
// up); their values meet in shared memory, where the epilogue warps take them up, so that the integer SiLU * up of one tile is
// evaluated under the multiplications of the next.
//
// Roles (27 or 31 warps): eight or sixteen read-out warps (lane = row, four or eight columns each), sixteen or eight expanding warps, one
// warp each for the MMAs, the TMA loads of planes and sums, and the bulk copies of packed weights (one super-block of 128 rows per copy slot); for gate / up four
// epilogue warps.  CTAs are
// persistent, one per SM, and walk the tiles of all groups, the column tiles of one weight slab next to each other.
// What bounds it: the instructions of all roles together, 6750 warp instructions per 128 x 256 weights at sixteen columns, a good part
// of them the hand-overs, at 2.3 to 2.7 per clock and SM; tensor pipe 12 % active at four rows an expert, 14 to 24 % at 2048 rows, HBM a
// quarter of its rate at most.  The forms of several digit counts share one allocation of registers: gate / up (64) and the dense product (72)
// spill, 1 % of the instructions.  One tile walks its super-blocks one behind the other, 1.3 us each: of a dense product with few tiles
// the CTAs of a cluster take a share of them each and join their sums through distributed shared memory (launch_tiles), calls of two and
// three rows are dispatched elsewhere (api.cu).
// Per block at 2048 tokens, in a profile: gate / up 880 us, down 583 (fully dequantised weights in four or five digits: 940, 1140); dense with the
// digits in front, 5120 x 2048: 2048 rows 277, 64 rows 23.5; at 64 tokens down 80 (warp-level MMAs 190; gate / up: tiles_few.cu).
// Every wait is bounded; on a time-out the CTA raises flag bit 3, leaves its loops, frees TMEM and exits.
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "layout.cuh"
#include "mma_items.cuh"
#include "tile_ops.cuh"

namespace iie {

__device__ unsigned long long d_tile_launches[TILE_SHAPES + TILE_FORMS];
__device__ int d_tile_form;                                        // gate / up of the call under way (tile_rows_kernel)

namespace {

constexpr int TL_WORK = 24;                                        // read-out and expanding warps
constexpr int TL_MMA_WARP = TL_WORK, TL_X_WARP = TL_MMA_WARP + 1, TL_W_WARP = TL_MMA_WARP + 2;
constexpr int TL_EPI = 4, TL_EPI_WARP = TL_W_WARP + 1;             // gate / up: warps that evaluate SiLU(g) * u
__host__ __device__ constexpr int tl_threads(int mode) { return (TL_EPI_WARP + (mode == MODE_GATEUP ? TL_EPI : 0)) * 32; }
constexpr int TL_MAX_STAGES = 4, TL_MAX_RAW = 3;
constexpr int TL_A_BYTES = 2 * 128 * 128;                          // two byte planes of 128 rows x 128 columns
constexpr int TL_MIN_SLOTS = 3;                                    // minima of three super-blocks, 128 rows x 32 columns each: the stages
constexpr int TL_MINS = TL_MIN_SLOTS * 128 * 32;                   // are at most two super-blocks ahead of the MMAs
constexpr int TL_EXCH = 16 * 128 * 8;                              // gate / up: sixteen columns of y on their way to the epilogue warps
constexpr int TL_SMEM = 217 * 1024;
constexpr int TL_MAX_GROUPS = 1024;
struct TileMaps { CUtensorMap x16, x32, s16, s32; };               // planes and sums, boxes of 16 and of 32 rows

// SPLIT: the CTAs of a cluster share the super-blocks of a tile (LINEAR; a form of its own: in one with the others it cost 2048 rows of a
// dense product 4 %)
template <int QT, int MODE, bool SPLIT>
__global__ void __launch_bounds__(tl_threads(MODE), 1) tile_kernel(const TileArgs a, const __grid_constant__ TileMaps maps) {
    constexpr bool Q4 = QT == QT_Q4K;
    constexpr int HTB = Q4 ? HTB_Q4K : HTB_Q6K, RAW_BYTES = 16 * HTB;
    constexpr int NROW = MODE == MODE_GATEUP ? 64 : 128;           // output rows of a tile
    extern __shared__ __align__(1024) unsigned char tl_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tl_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * TL_MAX_STAGES + 8 + 2 * TL_MAX_RAW + 3];
    __shared__ int s_first[TL_MAX_GROUPS + 1], s_off[TL_MAX_GROUPS + 1];       // first tile and first row of each group
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const uint32_t full_bar = tl_u32(bars), empty_bar = full_bar + 8 * TL_MAX_STAGES, acc_bar = empty_bar + 8 * TL_MAX_STAGES, free_bar = acc_bar + 8 * 4,
                   raw_full = free_bar + 8 * 4, raw_empty = raw_full + 8 * TL_MAX_RAW, y_full = raw_empty + 8 * TL_MAX_RAW, y_free = y_full + 8,
                   x_full = y_free + 8;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nb = a.nb;
    if (warp == TL_X_WARP && lane == 0) {                          // the tensor maps' first use would wait for them
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.x16)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.x32)) : "memory");
        if (Q4) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.s16)) : "memory");
        if (Q4) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&maps.s32)) : "memory");
    }
    if (MODE == MODE_GATEUP && a.few) {                            // tiles of eight rows may have the call
        pdl_enter();
        if (!*a.form) return;
    }
    if (warp == TL_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tl_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (MODE != MODE_GATEUP || !a.few) pdl_enter();                // what stands above needs nothing of the kernel before
    const int np = tl_planes(a.x_nl ? max(1, min(8, *a.x_nl)) : 8), ns = np + 1;        // uniform over the grid
    const bool wide = a.wide && (np == 3 || (!Q4 && (SPLIT ? np == 4 : a.wide == 2 && np <= 5)));      // (five digits beside the exchange: one stage)
    // Columns of a tile: 32 where the accumulators leave two TMEM buffers and the read-out's registers hold eight columns' sums: three planes, and
    // up to five of Q6_K, which has no minima (a weight is expanded half as often: a block of 2048 tokens, whose down projection has five digits,
    // 3208 -> 3050 us).
    const int bn = wide ? 32 : 16;
    const int n_rt = (int)((a.out_f + NROW - 1) / NROW);
    // CTAs that share a tile's super-blocks: those of a cluster, or of a half of it and so on where more digits than expected make the tiles
    // narrower and twice as many, so that no CTA walks two
    int split = SPLIT ? a.split : 1;
    if (SPLIT) while (split > 1 && (long long)split * ((a.n_rows + bn - 1) / bn) * n_rt > gridDim.x) split >>= 1;
    const int rank = SPLIT ? (int)(blockIdx.x & (split - 1)) : 0;
    // kept in shared memory: in registers they would push sums of the read-out out of theirs
    __shared__ int s_share[5];
    if (SPLIT && tid == 0) { s_share[0] = __ffs(split) - 1; s_share[1] = rank; s_share[2] = nb * rank / split; s_share[3] = nb * (rank + 1) / split; s_share[4] = (int)(blockIdx.x & (a.split - 1)) - rank; }
    auto share = [&](int i) { return *const_cast<const volatile int *>(&s_share[i]); };
    auto b_lo = [&] { return SPLIT ? share(2) : 0; };              // super-blocks of this CTA
    auto b_hi = [&] { return SPLIT ? share(3) : nb; };
    auto first_tile = [&] { return SPLIT ? (int)blockIdx.x >> share(0) : (int)blockIdx.x; };
    // The expansion bounds a tile of sixteen columns: sixteen of the warps expand there, as long as eight can hold the sums of the
    // read-out (eight columns a thread) in their registers
    const int n_read = wide || np > 5 ? 16 : 8, n_expand = TL_WORK - n_read;
    const bool thirds = Q4 && !wide;                               // the split of sc q, see above
    const int t_cols = (thirds ? 2 * np : np + 1) * bn, acc_cols = t_cols + (Q4 ? ns : 0) * bn;
    const int nbuf = min(4, 512 / acc_cols), buf_cols = acc_cols;
    const int x_bytes = np * bn * 128, s_bytes = Q4 ? ns * bn * 32 : 0;
    const int stage_bytes = (TL_A_BYTES + x_bytes + s_bytes + 1023) & ~1023;
    constexpr int FIXED = 1024 + (Q4 ? TL_MINS : 0) + (MODE == MODE_GATEUP ? TL_EXCH : 0);
    const int xch_bytes = SPLIT && split > 1 ? 128 * bn * 16 : 0;              // split tiles: sums of this CTA's share of the columns
    const int raw_slots = FIXED + xch_bytes + 3 * stage_bytes + TL_MAX_RAW * RAW_BYTES <= TL_SMEM ? TL_MAX_RAW : 2;
    const int stages = min(TL_MAX_STAGES, (TL_SMEM - FIXED - xch_bytes - raw_slots * RAW_BYTES) / stage_bytes);
    unsigned char *mins = smem + stages * stage_bytes, *exch = mins + (Q4 ? TL_MINS : 0), *raw = exch + (MODE == MODE_GATEUP ? TL_EXCH : xch_bytes);

    if (warp == 0) {                                               // first tile of every group
        int base = 0;
        for (int g0 = 0; g0 < a.n_groups; g0 += 32) {
            const int g = g0 + lane;
            const int at = g < a.n_groups && a.grp_off ? a.grp_off[g] : 0;
            const int rows = g < a.n_groups ? (a.grp_off ? a.grp_off[g + 1] - at : (int)a.n_rows) : 0;
            const int nt = (rows + bn - 1) / bn * n_rt;
            int incl = nt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, d); if (lane >= d) incl += t; }
            if (g < a.n_groups) { s_first[g] = base + incl - nt; s_off[g] = at; if (g + 1 == a.n_groups) s_off[g + 1] = at + rows; }
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_first[a.n_groups] = base;
    }
    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < TL_MAX_STAGES; s++) { tl_init(full_bar + 8 * s, n_expand + 1); tl_init(empty_bar + 8 * s, 1); }
        for (int s = 0; s < 4; s++) { tl_init(acc_bar + 8 * s, 1); tl_init(free_bar + 8 * s, n_read); }
        tl_init(y_full, n_read); tl_init(y_free, TL_EPI);
        tl_init(x_full, split * n_read);
        for (int s = 0; s < TL_MAX_RAW; s++) { tl_init(raw_full + 8 * s, 1); tl_init(raw_empty + 8 * s, TL_WORK); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (blockIdx.x == 0) {                                     // which tile shape ran (launch statistics)
            const int shape = Q4 && MODE == MODE_GATEUP ? (np == 3 ? 0 : np == 4 ? 1 : 7) : !Q4 && MODE == MODE_DOWN ? (np <= 5 ? 2 : np == 6 ? 3 : 7)
                              : Q4 && MODE == MODE_DOWN ? (np <= 5 ? 4 : 7) : Q4 && MODE == MODE_LINEAR ? (np == 3 ? 5 : np <= 5 ? 6 : 7) : 7;
            atomicAdd(&d_tile_launches[shape], 1ULL);
            if (SPLIT && split > 1) atomicAdd(&d_tile_launches[TILE_SHAPES], 1ULL);
            if (wide && np > 3) atomicAdd(&d_tile_launches[TILE_SHAPES + 1], 1ULL);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (SPLIT && split > 1) tl_cluster_sync();                     // the other CTAs' barriers stand
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    const int n_tiles = s_first[a.n_groups];
    auto next = [&](int tile) { return SPLIT ? n_tiles : tile + (int)gridDim.x; };       // (shared tiles: one per CTA)

    // tile -> group, row tile, first and past-the-last activation row
    struct Where { int g, rt, m0, m_end; };
    auto locate = [&](int tile) {
        int lo = 0, hi = a.n_groups;                               // s_first[lo] <= tile < s_first[hi]
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_first[mid] <= tile) lo = mid; else hi = mid; }
        const int first = s_off[lo], end = s_off[lo + 1], nt = (end - first + bn - 1) / bn, i = tile - s_first[lo];
        Where w;
        w.g = lo; w.rt = i / nt; w.m0 = first + (i - w.rt * nt) * bn; w.m_end = end;
        return w;
    };
    // weight units of half-tile `h` (0..15) of a tile
    const int n_ht = (int)((a.out_f + 7) >> 3);
    auto unit_of = [&](const Where &w, int h, const uint8_t *&p) {
        const int ht = MODE == MODE_GATEUP ? w.rt * 8 + (h & 7) : w.rt * 16 + h;
        const uint8_t *base = MODE == MODE_GATEUP && h >= 8 ? a.wb[w.g] : a.wa[w.g];
        p = base + (long long)ht * nb * HTB;
        return ht < n_ht;
    };

    if (warp < n_read) {
        // ================= read-out and epilogue ==============================================================
        const int rowt = (warp & 3) * 32 + lane, cg = warp >> 2;
        const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int meta_off = (rowt >> 3) * HTB + (Q4 ? 1024 + (rowt & 7) * 16 : 1664 + (rowt & 7) * 2);
        auto read_out = [&](auto np_c, auto bn_c, auto tpw_c) {
            constexpr int NP = decltype(np_c)::value, BN = decltype(bn_c)::value, TPW = decltype(tpw_c)::value, ROUNDS = TPW / 4;
            constexpr int NLV = (NP + 2) / 2;                      // 64-bit sums, 16 bits apart
            constexpr bool THIRDS = Q4 && BN == 16;
            constexpr int NT = THIRDS ? 2 * NP : NP + 1;           // accumulators of T
            TlRing rs, buf;
            uint32_t y_pass = 0;
            bool y_used = false;
            for (int tile = first_tile(); tile < n_tiles; tile = next(tile)) {
                const Where w = locate(tile);
                long long L[NLV][TPW];
#pragma unroll
                for (int i = 0; i < NLV; i++)
#pragma unroll
                    for (int j = 0; j < TPW; j++) L[i][j] = 0;
                bool ok = true;
                for (int b = b_lo(); b < b_hi(); b++) {
                    if (!(ok = tl_wait(raw_full + 8 * rs.slot, rs.pass, &s_abort))) break;
                    const unsigned char *meta = raw + rs.slot * RAW_BYTES + meta_off;
                    int d, dm = 0;
                    if (Q4) {
                        const uint32_t h = *reinterpret_cast<const uint32_t *>(meta);
                        d = scale_small(h & 0xFFFF, a.fw); dm = (THIRDS ? -1 : -16) * scale_small(h >> 16, a.fw);
                    } else d = scale_small(*reinterpret_cast<const unsigned short *>(meta), a.fw);
                    const int d8 = d << 8;
                    __syncwarp();
                    if (lane == 0) tl_arrive(raw_empty + 8 * rs.slot);
                    if (!(ok = tl_wait(acc_bar + 8 * buf.slot, buf.pass, &s_abort))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t base = tlane + buf.slot * buf_cols + cg * TPW;
#pragma unroll
                    for (int ro = 0; ro < ROUNDS; ro++) {
                        if (THIRDS) {                              // two digits at a time: what the registers hold
#pragma unroll
                            for (int s0 = 0; s0 < NP; s0 += 2) {
                                int r[2][2][4];
#pragma unroll
                                for (int s = s0; s < s0 + 2 && s < NP; s++) { tl_ld4(base + s * BN + ro * 4, r[s - s0][0]); tl_ld4(base + (NP + s) * BN + ro * 4, r[s - s0][1]); }
                                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                                for (int s = s0; s < s0 + 2 && s < NP; s++)
#pragma unroll
                                    for (int j = 0; j < 4; j++) L[s / 2][ro * 4 + j] += (long long)(r[s - s0][0][j] + 8 * r[s - s0][1][j]) * (long long)((s & 1) ? d8 : d);
                            }
                        } else {
                            int r[NT][4];
#pragma unroll
                            for (int s = 0; s < NT; s++) tl_ld4(base + s * BN + ro * 4, r[s]);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int s = 0; s < NT; s++)
#pragma unroll
                                for (int j = 0; j < 4; j++) L[s / 2][ro * 4 + j] += (long long)r[s][j] * (long long)((s & 1) ? d8 : d);
                        }
                        if (Q4) {
                            int r[NP + 1][4];
#pragma unroll
                            for (int s = 0; s <= NP; s++) tl_ld4(base + (NT + s) * BN + ro * 4, r[s]);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int s = 0; s <= NP; s += 2)
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const int m = r[s][j] + (s + 1 <= NP ? r[s + 1 <= NP ? s + 1 : s][j] * 256 : 0);     // < 2^27
                                    L[s / 2][ro * 4 + j] += (long long)m * (long long)dm;
                                }
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tl_arrive(free_bar + 8 * buf.slot);
                    rs.step(raw_slots); buf.step(nbuf);
                }
                if (!ok) break;
                // ---- y = floor(V / 2^fw), then what the product is for ---------------------------------------
                const int sh = a.fw + (Q4 && !THIRDS ? 4 : 0);
                if (SPLIT && share(0) > 0) {
                    // column c of the tile belongs to CTA c mod split, as its column c / split there: everybody's sums go to the owner in 128
                    // bits, which adds them up and stores
#pragma unroll
                    for (int j = 0; j < TPW; j++) {
                        const int c = cg * TPW + j, ls = share(0);
                        i128 v = L[NLV - 1][j];
#pragma unroll
                        for (int i = NLV - 2; i >= 0; i--) v = (v << 16) + (i128)L[i][j];
                        tl_remote_store(tl_remote(tl_u32(exch) + (uint32_t)((share(1) * (BN >> ls) + (c >> ls)) * 128 + rowt) * 16, share(4) + (c & ((1 << ls) - 1))), v);
                    }
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    __syncwarp();
                    const int ls = share(0), split = 1 << ls, cols = BN >> ls;   // columns of this CTA
                    if (lane < split) tl_remote_arrive(tl_remote(x_full, share(4) + lane));
                    if (!(ok = tl_wait_cluster(x_full, 0, &s_abort))) break;      // (one tile per CTA: the barrier's only phase)
                    const long long row = (long long)w.rt * 128 + rowt;
#pragma unroll 1                                                   // (unrolled, these two cost the whole read-out registers)
                    for (int slot = cg; slot < cols; slot += n_read / 4) {
                        const ulonglong2 *from = reinterpret_cast<const ulonglong2 *>(exch) + slot * 128 + rowt;
                        i128 v = 0;
#pragma unroll 1
                        for (int k = 0; k < split; k++, from += cols * 128) { const ulonglong2 p = *from; v += (i128)(((u128)p.y << 64) | p.x); }
                        const int colx = w.m0 + slot * split + share(1);
                        if (row < a.out_f && colx < w.m_end) a.out[(long long)colx * a.out_f + row] = (long long)(v >> sh);
                    }
                    continue;
                }
                long long y[TPW];
#pragma unroll
                for (int j = 0; j < TPW; j++) {
                    i128 v = L[NLV - 1][j];
#pragma unroll
                    for (int i = NLV - 2; i >= 0; i--) v = (v << 16) + (i128)L[i][j];
                    y[j] = (long long)(v >> sh);
                }
                const int col0 = w.m0 + cg * TPW;
                if (MODE == MODE_GATEUP) {
                    // sixteen columns of the tile at a time to the epilogue warps
                    constexpr int PER = BN == 32 ? 4 : TPW;        // of this thread
                    long long *to = reinterpret_cast<long long *>(exch) + cg * PER * 128 + rowt;
#pragma unroll
                    for (int q = 0; q < TPW; q += PER) {
                        if (y_used && !(ok = tl_wait(y_free, y_pass ^ 1, &s_abort))) break;
#pragma unroll
                        for (int j = 0; j < PER; j++) to[j * 128] = y[q + j];
                        __syncwarp();
                        if (lane == 0) tl_arrive(y_full);
                        y_used = true; y_pass ^= 1;
                    }
                    if (!ok) break;
                } else {
                    const long long row = (long long)w.rt * 128 + rowt;
                    if (row < a.out_f) {
#pragma unroll
                        for (int j = 0; j < TPW; j++) {
                            const int colx = col0 + j;
                            if (colx >= w.m_end) continue;
                            if (MODE == MODE_LINEAR) a.out[(long long)colx * a.out_f + row] = y[j];
                            else {
                                const long long tok = a.pair_tok ? a.pair_tok[colx] : colx;
                                atomicAdd(reinterpret_cast<unsigned long long *>(a.out + tok * a.out_f + row), (unsigned long long)mul_shift(y[j], a.gates[colx], a.fa));
                            }
                        }
                    }
                }
            }
        };
        using std::integral_constant;
        if (!Q4 && wide && np == 4) read_out(integral_constant<int, Q4 ? 3 : 4>{}, integral_constant<int, 32>{}, integral_constant<int, 8>{});
        else if (!Q4 && wide && np == 5) read_out(integral_constant<int, Q4 ? 3 : 5>{}, integral_constant<int, 32>{}, integral_constant<int, 8>{});
        else if (np == 3 && wide) read_out(integral_constant<int, 3>{}, integral_constant<int, 32>{}, integral_constant<int, 8>{});
        else if (np == 3) read_out(integral_constant<int, 3>{}, integral_constant<int, 16>{}, integral_constant<int, 8>{});
        else if (np == 4) read_out(integral_constant<int, 4>{}, integral_constant<int, 16>{}, integral_constant<int, 8>{});
        else if (np == 5) read_out(integral_constant<int, 5>{}, integral_constant<int, 16>{}, integral_constant<int, 8>{});
        else if (np == 6) read_out(integral_constant<int, 6>{}, integral_constant<int, 16>{}, integral_constant<int, 4>{});
        else read_out(integral_constant<int, 8>{}, integral_constant<int, 16>{}, integral_constant<int, 4>{});
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp < TL_MMA_WARP) {
        // ================= expansion: packed codes -> the two bytes of sc * q, half a super-block per stage ============
        const int ew = warp - n_read, g = lane >> 2, t = lane & 3;         // half-tiles ew, ew + n_expand; row g, quarter t of a unit
        // Q4_K: sub-block m of the half (columns 32 m ..): this lane's eight bytes are half of 16-byte chunk 2 m + (t >> 1).  Lanes of
        // odd g take their two groups in the other order, so that the 16 lanes of a store phase fall on all banks.
        // Q6_K: word (kq, u) is byte 4 t of chunk 2 kq + u: eight rows, eight chunks, all banks.
        uint32_t off[8];
#pragma unroll
        for (int i = 0; i < (Q4 ? 4 : 8); i++)
            off[i] = (uint32_t)(g * 128) + (Q4 ? ((((2 * (i ^ (2 * (g & 1))) + (t >> 1)) ^ g) << 4) + (t & 1) * 8) : (((i ^ g) << 4) + 4 * t));
        auto expand = [&](auto nh_c, auto th_c) {
        constexpr int NH = decltype(nh_c)::value;                  // half-tiles of a warp
        constexpr bool THIRDS = decltype(th_c)::value;
        TlRing rs, st;
        int n_mins = 0;
        bool ok = true;
        for (int tile = first_tile(); tile < n_tiles && ok; tile = next(tile)) {
            for (int b = b_lo(); b < b_hi() && ok; b++) {
                if (!(ok = tl_wait(raw_full + 8 * rs.slot, rs.pass, &s_abort))) break;
                const unsigned char *slot = raw + rs.slot * RAW_BYTES;
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    // this lane's share of the two half-tiles, before the wait for the stage
                    uint4 q_in[NH], meta_in[NH];
                    uint2 hw_in[NH], sc_in[NH];
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        const unsigned char *unit = slot + (ew + n_expand * h) * HTB;
                        q_in[h] = *reinterpret_cast<const uint4 *>(unit + p * 512 + lane * 16);
                        if (Q4) meta_in[h] = *reinterpret_cast<const uint4 *>(unit + 1024 + g * 16);
                        else {
                            hw_in[h] = *reinterpret_cast<const uint2 *>(unit + 1024 + lane * 16 + p * 8);                  // high bits of u0, u1
                            sc_in[h] = *reinterpret_cast<const uint2 *>(unit + 1536 + g * 16 + p * 8);                     // int8 scale of (kq, u) at byte 2 kq + u
                        }
                    }
                    if (st.lapped && !(ok = tl_wait(empty_bar + 8 * st.slot, st.pass ^ 1, &s_abort))) break;
                    const uint32_t dst = tl_u32(smem + st.slot * stage_bytes);
#pragma unroll
                    for (int h = 0; h < NH; h++) {
                        const uint32_t to = dst + (ew + n_expand * h) * 1024;           // eight rows of 128 bytes
                        if (Q4) {
                            uint4 q = q_in[h];
                            const uint4 meta = meta_in[h];
                            uint32_t sc[2], mn[2];
                            q4k_scales(meta.y, meta.z, meta.w, sc[0], sc[1], mn[0], mn[1]);
                            uint32_t scw = p ? sc[1] : sc[0];
                            if (g & 1) { q = make_uint4(q.z, q.w, q.x, q.y); scw = __byte_perm(scw, 0, 0x1032); }
                            const uint32_t sc_lo = scw & 0x07070707u, sc_hi = (scw >> 3) & 0x07070707u;
                            if (p == 0) {                          // the row's eight minima, in the columns of this super-block's sums
                                const int r = (ew + n_expand * h) * 8 + g;
                                const bool mine = t == (b & 3);
                                tl_sts64(tl_u32(mins) + n_mins * (128 * 32) + r * 32 + (((t >> 1) ^ ((r >> 2) & 1)) << 4) + (t & 1) * 8, mine ? mn[0] : 0, mine ? mn[1] : 0);
                            }
#pragma unroll
                            for (int i = 0; i < 2; i++) {          // group: low nibbles sub-block 2 i, high nibbles 2 i + 1
                                const uint32_t w0 = i ? q.z : q.x, w1 = i ? q.w : q.y;
                                if (THIRDS) {                      // sixteen columns: sc = 8 sh + sl, four products below 106 per multiplication
#pragma unroll
                                    for (int nib = 0; nib < 2; nib++) {
                                        const uint32_t x0 = (nib ? w0 >> 4 : w0) & 0x0f0f0f0fu, x1 = (nib ? w1 >> 4 : w1) & 0x0f0f0f0fu;
                                        const uint32_t sl = (uint32_t)ubyte_at(sc_lo, 2 * i + nib), sh = (uint32_t)ubyte_at(sc_hi, 2 * i + nib);
                                        tl_sts64(to + off[2 * i + nib], x0 * sl, x1 * sl);
                                        tl_sts64(to + off[2 * i + nib] + TL_A_BYTES / 2, x0 * sh, x1 * sh);
                                    }
                                    continue;
                                }
                                const uint32_t v0 = w0 >> 8, v1 = w1 >> 8;
                                const uint32_t s0 = (uint32_t)ubyte_at(scw, 2 * i) * 16, s1 = (uint32_t)ubyte_at(scw, 2 * i + 1);
                                // two 16-bit products per multiplication; 16 sc q in both halves of a byte
                                const uint32_t a0 = (w0 & 0x000f000fu) * s0, a1 = (v0 & 0x000f000fu) * s0, b0 = (w1 & 0x000f000fu) * s0, b1 = (v1 & 0x000f000fu) * s0;
                                tl_sts64(to + off[2 * i], __byte_perm(a0, a1, 0x6240), __byte_perm(b0, b1, 0x6240));
                                tl_sts64(to + off[2 * i] + TL_A_BYTES / 2, __byte_perm(a0, a1, 0x7351), __byte_perm(b0, b1, 0x7351));
                                const uint32_t c0 = (w0 & 0x00f000f0u) * s1, c1 = (v0 & 0x00f000f0u) * s1, e0 = (w1 & 0x00f000f0u) * s1, e1 = (v1 & 0x00f000f0u) * s1;
                                tl_sts64(to + off[2 * i + 1], __byte_perm(c0, c1, 0x6240), __byte_perm(e0, e1, 0x6240));
                                tl_sts64(to + off[2 * i + 1] + TL_A_BYTES / 2, __byte_perm(c0, c1, 0x7351), __byte_perm(e0, e1, 0x7351));
                            }
                        } else {
                            const uint4 lw = q_in[h];              // low nibbles, u0: {first, second 32}, u1: {..}
                            const uint2 hw = hw_in[h], scs = sc_in[h];
#pragma unroll
                            for (int kq = 0; kq < 4; kq++)
#pragma unroll
                                for (int u = 0; u < 2; u++) {
                                    const uint32_t n = (kq & 1) ? (u ? lw.w : lw.y) : (u ? lw.z : lw.x), hb = u ? hw.y : hw.x;
                                    const uint32_t hs = kq == 0 ? hb << 4 : kq == 1 ? hb << 2 : kq == 2 ? hb : hb >> 2;
                                    const uint32_t q = ((kq < 2 ? n : n >> 4) & 0x0f0f0f0fu) | (hs & 0x30303030u);
                                    const int sc = sbyte_at(kq < 2 ? scs.x : scs.y, 2 * (kq & 1) + u);
                                    // (q - 32) sc + 2^15 in both 16-bit halves: no borrow between them
                                    const uint32_t bias = 0x80008000u - 0x00200020u * (uint32_t)sc;
                                    const uint32_t e = __byte_perm(q, 0, 0x4240) * (uint32_t)sc + bias, o = __byte_perm(q, 0, 0x4341) * (uint32_t)sc + bias;
                                    tl_sts32(to + off[2 * kq + u], __byte_perm(e, o, 0x6240));
                                    tl_sts32(to + off[2 * kq + u] + TL_A_BYTES / 2, __byte_perm(e, o, 0x7351) ^ 0x80808080u);
                                }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tl_arrive(full_bar + 8 * st.slot);
                        if (p == 1) tl_arrive(raw_empty + 8 * rs.slot);
                    }
                    st.step(stages);
                }
                rs.step(raw_slots);
                n_mins = n_mins + 1 == TL_MIN_SLOTS ? 0 : n_mins + 1;
            }
        }
        };
        using std::integral_constant;
        if (n_expand == 16) expand(integral_constant<int, 1>{}, integral_constant<bool, Q4>{});
        else if (thirds) expand(integral_constant<int, 2>{}, integral_constant<bool, Q4>{});
        else expand(integral_constant<int, 2>{}, integral_constant<bool, false>{});
    } else if (warp == TL_MMA_WARP) {
        // ================= MMAs (the whole warp walks the loop, one elected lane issues) ===============================
        const uint32_t leader = tl_elect();
        const uint32_t id_lo = tl_idesc(np * bn, false), id_hi = tl_idesc(np * bn, !Q4), id_first = tl_idesc(bn, false), id_rest = tl_idesc((np - 1) * bn, false),
                       id_min = tl_idesc(ns * bn, false);
        TlRing st, buf;
        int n_mins = 0;
        bool ok = true;
        for (int tile = first_tile(); tile < n_tiles && ok; tile = next(tile))
            for (int b = b_lo(); b < b_hi() && ok; b++) {
                if (buf.lapped && !(ok = tl_wait(free_bar + 8 * buf.slot, buf.pass ^ 1, &s_abort))) break;
                const uint32_t d = tmem + buf.slot * buf_cols;
                for (int p = 0; p < 2; p++) {
                    if (!(ok = tl_wait(full_bar + 8 * st.slot, st.pass, &s_abort))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t stage = tl_u32(smem + st.slot * stage_bytes);
                    const uint64_t lo = tl_desc128(stage), hi = tl_desc128(stage + TL_A_BYTES / 2), x = tl_desc128(stage + TL_A_BYTES);
                    if (leader) {
#pragma unroll
                        for (int ks = 0; ks < 4; ks++) {
                            if (thirds) {
                                tl_mma(d, lo + ks * 2, x + ks * 2, id_lo, p | ks);
                                tl_mma(d + np * bn, hi + ks * 2, x + ks * 2, id_lo, p | ks);
                            } else if (p == 0 && ks == 0) {        // the high bytes open columns bn.., the first plane of the low bytes columns 0..
                                tl_mma(d + bn, hi, x, id_hi, 0);
                                tl_mma(d, lo, x, id_first, 0);
                                tl_mma(d + bn, lo, x + bn * 8, id_rest, 1);
                            } else {
                                tl_mma(d, lo + ks * 2, x + ks * 2, id_lo, 1);
                                tl_mma(d + bn, hi + ks * 2, x + ks * 2, id_hi, 1);
                            }
                        }
                        if (Q4 && p == 0) tl_mma(d + t_cols, tl_desc32(tl_u32(mins) + n_mins * (128 * 32)), tl_desc32(stage + TL_A_BYTES + x_bytes), id_min, 0);
                        tl_commit(empty_bar + 8 * st.slot);
                        if (p == 1) tl_commit(acc_bar + 8 * buf.slot);
                    }
                    __syncwarp();
                    st.step(stages);
                }
                buf.step(nbuf);
                n_mins = n_mins + 1 == TL_MIN_SLOTS ? 0 : n_mins + 1;
            }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    } else if (warp == TL_X_WARP) {
        // ================= digit planes and sub-block sums of the tile's rows ==================================
        if (lane == 0) {
            const CUtensorMap *xm = wide ? &maps.x32 : &maps.x16, *sm = wide ? &maps.s32 : &maps.s16;
            TlRing st;
            bool ok = true;
            for (int tile = first_tile(); tile < n_tiles && ok; tile = next(tile)) {
                const Where w = locate(tile);
                for (int c = 2 * b_lo(); c < 2 * b_hi(); c++) {
                    const uint32_t eb = empty_bar + 8 * st.slot, fb = full_bar + 8 * st.slot;
                    if (st.lapped && !(ok = tl_try(eb, st.pass ^ 1) || tl_wait_slow(eb, st.pass ^ 1, &s_abort))) break;
                    const uint32_t dst = tl_u32(smem + st.slot * stage_bytes + TL_A_BYTES);
                    const bool sums = Q4 && (c & 1) == 0;
                    tl_expect(fb, x_bytes + (sums ? s_bytes : 0));
                    for (int l = 0; l < np; l++) tl_tma(dst + l * bn * 128, xm, c * 128, l, w.m0, fb);
                    if (sums) for (int l = 0; l < ns; l++) tl_tma(dst + x_bytes + l * bn * 32, sm, (c >> 3) * 32, l, w.m0, fb);
                    st.step(stages);
                }
            }
            // given up: the copies in flight land before the CTA leaves (a slot behind the ring's position is in its current lap)
            if (!ok) for (int s = 0; s < stages; s++)
                for (unsigned it = 0; it < TL_WAIT_LIMIT && !tl_try(full_bar + 8 * s, s < st.slot ? st.pass : st.pass ^ 1); it++) {}
        }
    } else if (warp == TL_W_WARP) {
        // ================= packed weights: one super-block of the tile's 16 half-tiles per slot ===============
        TlRing rs;
        bool ok = true;
        for (int tile = first_tile(); tile < n_tiles && ok; tile = next(tile)) {
            const Where w = locate(tile);
            const uint8_t *src = nullptr;
            const bool live = lane < 16 && unit_of(w, lane, src);
            const int n_live = __popc(__ballot_sync(0xffffffffu, live));
            for (int b = b_lo(); b < b_hi(); b++) {
                const uint32_t eb = raw_empty + 8 * rs.slot, fb = raw_full + 8 * rs.slot;
                if (rs.lapped && !(ok = tl_wait(eb, rs.pass ^ 1, &s_abort))) break;
                if (lane == 0) tl_expect(fb, n_live * HTB);
                __syncwarp();
                if (live) asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                       ::"r"(tl_u32(raw + rs.slot * RAW_BYTES + lane * HTB)), "l"(src + (long long)b * HTB), "r"(HTB), "r"(fb) : "memory");
                rs.step(raw_slots);
            }
        }
        if (!ok && lane == 0) for (int s = 0; s < raw_slots; s++)
            for (unsigned it = 0; it < TL_WAIT_LIMIT && !tl_try(raw_full + 8 * s, s < rs.slot ? rs.pass : rs.pass ^ 1); it++) {}
    } else if (MODE == MODE_GATEUP) {
        // ================= epilogue of gate / up: SiLU(g) * u and its digit planes =============================
        const int et = tid - TL_EPI_WARP * 32, r = et & 63, half = et >> 6;      // output row of the tile, odd or even columns
        int nl_max = 0;
        uint32_t pass = 0;
        bool ok = true;
        for (int tile = first_tile(); tile < n_tiles && ok; tile = next(tile)) {
            const Where w = locate(tile);
            const long long row = (long long)w.rt * 64 + r;
            for (int q = 0; q < bn / 4; q += 4) {                  // wide: columns 8 g + q + (0..3) of column group g = 0..3
                if (!(ok = tl_wait(y_full, pass, &s_abort))) break;
                const long long *from = reinterpret_cast<const long long *>(exch) + half * 128 + r;
                int64_t gu[8];
                bool least = false;
#pragma unroll
                for (int i = 0; i < 8; i++) {                      // every column, live or not: the chains interleave
                    const int64_t g = from[2 * i * 128];
                    least |= g == INT64_MIN;
                    gu[i] = silu_up_fixed(g, from[2 * i * 128 + 64], a.fa, a.sig_log2e, a.sig_clip);
                }
                if (least)
#pragma unroll
                    for (int i = 0; i < 8; i++) gu[i] = silu_up_any(from[2 * i * 128], from[2 * i * 128 + 64], a.fa, a.sig_log2e, a.sig_clip);
                __syncwarp();
                if (lane == 0) tl_arrive(y_free);
                pass ^= 1;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int c = 2 * i + half, col = w.m0 + (wide ? (c >> 2) * 8 + q + (c & 3) : c);
                    if (col >= w.m_end || row >= a.out_f) continue;
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
        }
        if (a.out_nl) {
            nl_max = __reduce_max_sync(0xffffffffu, nl_max);
            if (lane == 0 && nl_max > 0) atomicMax(a.out_nl, nl_max);
        }
    }
    __syncthreads();
    if (SPLIT && share(0) > 0) tl_cluster_sync();                  // nobody leaves while another CTA stores or arrives here
    if (warp == TL_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
    if (tid == 0 && s_abort) atomicOr(a.flags, 8);
}

// Sums of the 32 columns of every sub-block as nine balanced digits, xs[row][9][stride] (columns from nb * 8 on are zero), and with
// `xidx` the digit planes in use copied into pair order.  One thread per (row, sub-block).
// With `form` the last block says which tiles of gate / up take the rows: 1 of sixteen, 0 of eight.
__global__ void __launch_bounds__(256) tile_rows_kernel(const int8_t *xl, const int *xidx, const int *n_live, const int *x_nl,
                                                        long long n_rows, int nb, int stride, int8_t *xg, int8_t *xs, const int *grp_off, int n_groups, int n_rt, int *form) {
    pdl_enter();
    if (form && blockIdx.x == gridDim.x - 1) {
        int of8 = 0, of16 = 0;
        if (threadIdx.x >= 32) return;
        for (int g = threadIdx.x; g < n_groups; g += 32) { const int rows = grp_off[g + 1] - grp_off[g]; of8 += (rows + 7) / 8; of16 += (rows + 15) / 16; }
        of8 = __reduce_add_sync(0xffffffffu, of8); of16 = __reduce_add_sync(0xffffffffu, of16);
        if (threadIdx.x == 0) *form = tl_rows_of_sixteen((long long)of8 * n_rt, (long long)of16 * n_rt) ? 1 : 0;
        return;
    }
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    const int j = (int)(idx % stride);
    const long long row = idx / stride;
    if (row >= n_rows || (n_live && row >= *n_live)) return;
    const int np = tl_planes(x_nl ? max(1, min(8, *x_nl)) : 8);
    const long long K = (long long)nb * 256;
    int8_t *to = xs ? xs + row * 9 * stride + j : nullptr;
    if (j >= nb * 8) {
        if (to) for (int l = 0; l < 9; l++) to[l * stride] = 0;
        return;
    }
    const int8_t *src = xl + (xidx ? (long long)xidx[row] : row) * 8 * K + j * 32;
    int carry = 0;
    for (int l = 0; l < 9; l++) {
        if (l < np) {
            const uint4 u = __ldcg(reinterpret_cast<const uint4 *>(src + l * K)), v = __ldcg(reinterpret_cast<const uint4 *>(src + l * K + 16));
            if (xidx) {
                uint4 *dst = reinterpret_cast<uint4 *>(xg + row * 8 * K + l * K + j * 32);
                dst[0] = u; dst[1] = v;
            }
            carry = __dp4a((int)u.x, 0x01010101, carry); carry = __dp4a((int)u.y, 0x01010101, carry);
            carry = __dp4a((int)u.z, 0x01010101, carry); carry = __dp4a((int)u.w, 0x01010101, carry);
            carry = __dp4a((int)v.x, 0x01010101, carry); carry = __dp4a((int)v.y, 0x01010101, carry);
            carry = __dp4a((int)v.z, 0x01010101, carry); carry = __dp4a((int)v.w, 0x01010101, carry);
        }
        const int d = (int)(int8_t)carry;                          // digit in [-128, 127], the rest is a multiple of 256
        if (to) to[l * stride] = (int8_t)d;
        carry = (carry - d) >> 8;
    }
}

template <int QT, int MODE, bool SPLIT>
cudaError_t launch_tile(const TileArgs &a, const TileMaps &maps, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(tile_kernel<QT, MODE, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TL_SMEM);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    const long long n_rt = (a.out_f + (MODE == MODE_GATEUP ? 63 : 127)) / (MODE == MODE_GATEUP ? 64 : 128);
    if (SPLIT) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(a.split * ((a.n_rows + (a.wide ? 31 : 15)) / (a.wide ? 32 : 16)) * n_rt));
        cfg.blockDim = dim3(tl_threads(MODE)); cfg.dynamicSmemBytes = TL_SMEM; cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = (unsigned)a.split; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 2;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, tile_kernel<QT, MODE, SPLIT>, a, maps);
        note_launch();
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    // an upper bound on the tiles: every group may end in a partial one
    const long long most = (a.n_rows / 16 + std::min<long long>(a.n_groups, a.n_rows)) * n_rt;
    launch_behind(tile_kernel<QT, MODE, SPLIT>, (unsigned)std::max<long long>(1, std::min<long long>(148, most)), tl_threads(MODE), TL_SMEM, s, a, maps);
    note_launch();
    return cudaGetLastError();
}

}  // namespace

size_t tile_sums_bytes(long long rows, long long n_blocks) { return (size_t)rows * 9 * (size_t)((n_blocks * 8 + 31) / 32 * 32); }

cudaError_t launch_tiles(int qtype, int mode, const TileArgs &args, cudaStream_t s) {
    TileArgs a = args;
    if (a.nb <= 0 || a.nb > 64 || a.n_groups <= 0 || a.n_groups > TL_MAX_GROUPS || a.out_f <= 0 || a.n_rows <= 0 || a.n_rows > (1 << 28) || (!a.grp_off && a.n_groups != 1) ||
        (reinterpret_cast<uintptr_t>(a.xl) & 15) || (a.xidx && !a.xg) || !tl_encode()) return cudaErrorNotSupported;
    if (qtype != QT_Q4K && !(qtype == QT_Q6K && mode != MODE_GATEUP)) return cudaErrorNotSupported;
    if (qtype == QT_Q4K && !a.xs) return cudaErrorInvalidValue;
    a.sig_log2e = sigmoid_log2e(a.fa); a.sig_clip = sigmoid_clip(a.fa);
    // Sixteen columns while a group has few rows: a 32-column tile would multiply mostly padding.  A 32-column tile of four and five digits takes
    // a fifth longer than one of sixteen, so it also wants more narrow tiles than one wave (Q6_K, five digits: 5120 x 2048, 33 rows, 120 narrow
    // tiles 19.8 us against 24.0; 64 rows, 160 narrow tiles 33.8 against 25.4; 9216 x 4096, 100 rows 104 against 72.5) and groups that fill more
    // than one (blocks of 128 experts with 14 / 16 / 20 / 24 / 32 rows each 410 / 427 / 469 / 516 / 620 us narrow, 415 / 434 / 475 / 508 / 605 wide).
    a.wide = a.n_rows > 12LL * a.n_groups && a.n_rows > 16;
    if (a.wide && a.n_rows > (a.grp_off ? 20LL * a.n_groups : 0) && (a.n_rows + 15) / 16 * ((a.out_f + 127) / 128) > 148) a.wide = 2;
    // A matrix of few tiles: clusters of CTAs share a tile's super-blocks, as long as all clusters fit on the device at once (one CTA per
    // SM; 33 clusters of four, 15 of eight) and the walk gets shorter by more than the clusters cost.  A super-block is 1.2 to 1.7 us of a
    // tile's walk; the launch of clusters and the exchange are 3.5 us (Q4_K) to 5.  Q4_K, 7 rows: 128 x 2048 19.8 -> 13 us, 5120 x 2048 20.2
    // -> 16.9, 2048 x 4096 30.4 -> 16.9, three super-blocks saved 1024 x 1024 14.8 -> 12.9, one saved 2048 x 768 13.6 -> 14.9; 64 rows: 2048 x
    // 2048 23.2 -> 19.4, 2048 x 4096 36.2 -> 23.4.  Q6_K, 7 rows: 5120 x 2048 (four saved) 17.9 -> 16.5, 1024 x 1024 (three) 12.6 -> 12.3; 64 rows:
    // 2048 x 2048 21.3 -> 18.0, 100 rows (four) 22.7 -> 21.5.  With more digits than three the tiles of 17 rows and more are narrower, and half as
    // many CTAs share one: that is 10 % and more faster, too (Q4_K 2048 x 4096, 64 rows, four digits 35.2 -> 27.9), or as fast but for Q6_K of
    // five digits and more where nobody shares (4096 x 4096, 40 rows 31.2 -> 33.9 us, and 20.1 -> 22.5 were four saved enough).
    a.split = 1;
    const bool q4 = qtype == QT_Q4K;
    const long long whole = ((a.n_rows + (a.wide ? 31 : 15)) / (a.wide ? 32 : 16)) * ((a.out_f + 127) / 128);
    while (mode == MODE_LINEAR && a.split < 8 && 2 * a.split <= a.nb && whole <= (a.split == 1 ? 74 : a.split == 2 ? 33 : 15)) a.split *= 2;
    if (a.nb - (a.nb + a.split - 1) / a.split < (q4 ? 3 : a.wide ? 6 : 4)) a.split = 1;
    const int stride = (a.nb * 8 + 31) / 32 * 32;
    // Gate / up by tiles of eight rows, and by those of sixteen beside them where the rows may lie on so few experts that these are quicker
    // (tl_rows_of_sixteen): the kernel in front finds out for both; the launch that has nothing to do costs 1.5 us.
    a.few = !a.few || !q4 || mode != MODE_GATEUP || !a.grp_off ? 0 : a.n_rows * ((a.out_f + 63) / 64) > 16LL * TL_SIXTEEN_FROM ? 2 : 1;
    if (a.few) {
        void *counts = nullptr, *form = nullptr;
        if (cudaGetSymbolAddress(&counts, d_tile_launches) != cudaSuccess || cudaGetSymbolAddress(&form, d_tile_form) != cudaSuccess) return cudaErrorInvalidValue;
        a.counts = static_cast<unsigned long long *>(counts); a.form = static_cast<int *>(form);
        a.wide = 0;
    }
    if ((q4 && !a.xs_ready) || a.xidx) {
        const long long n = a.n_rows * stride;
        launch_behind(tile_rows_kernel, (unsigned)((n + 255) / 256 + (a.few == 2)), 256, 0, s, a.xl, a.xidx, a.grp_off ? a.grp_off + a.n_groups : nullptr, a.x_nl, a.n_rows, a.nb, stride, a.xg, q4 ? a.xs : nullptr,
                      a.grp_off, a.n_groups, (int)((a.out_f + 63) / 64), a.few == 2 ? a.form : nullptr);
        note_launch();
    } else if (a.few) a.few = 1;
    const int8_t *x = a.xidx ? a.xg : a.xl;
    if (a.few) {
        const cudaError_t e = launch_tiles_few(a, x, s);
        if (e != cudaSuccess || a.few == 1) return e;
    }
    TileMaps maps;
    const long long K = (long long)a.nb * 256;
    bool ok = tl_map(&maps.x16, x, K, 8, a.n_rows, 128, 16, CU_TENSOR_MAP_SWIZZLE_128B) && tl_map(&maps.x32, x, K, 8, a.n_rows, 128, 32, CU_TENSOR_MAP_SWIZZLE_128B);
    if (q4) ok = ok && tl_map(&maps.s16, a.xs, stride, 9, a.n_rows, 32, 16, CU_TENSOR_MAP_SWIZZLE_32B) && tl_map(&maps.s32, a.xs, stride, 9, a.n_rows, 32, 32, CU_TENSOR_MAP_SWIZZLE_32B);
    else maps.s16 = maps.s32 = maps.x16;
    if (!ok) return cudaErrorInvalidValue;
    if (a.split > 1) return q4 ? launch_tile<QT_Q4K, MODE_LINEAR, true>(a, maps, s) : launch_tile<QT_Q6K, MODE_LINEAR, true>(a, maps, s);
    if (q4 && mode == MODE_LINEAR) return launch_tile<QT_Q4K, MODE_LINEAR, false>(a, maps, s);
    if (q4 && mode == MODE_GATEUP) return launch_tile<QT_Q4K, MODE_GATEUP, false>(a, maps, s);
    if (q4) return launch_tile<QT_Q4K, MODE_DOWN, false>(a, maps, s);
    if (mode == MODE_LINEAR) return launch_tile<QT_Q6K, MODE_LINEAR, false>(a, maps, s);
    return launch_tile<QT_Q6K, MODE_DOWN, false>(a, maps, s);
}

void tile_launch_counts(unsigned long long *out) {
    if (cudaMemcpyFromSymbol(out, d_tile_launches, sizeof(unsigned long long) * (TILE_SHAPES + TILE_FORMS)) != cudaSuccess) {
        cudaGetLastError();
        for (int i = 0; i < TILE_SHAPES + TILE_FORMS; i++) out[i] = 0;
    }
}

}  // namespace iie
