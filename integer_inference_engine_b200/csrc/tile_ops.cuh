// What the tcgen05 tiles of tiles.cu and tiles_few.cu share: barriers with bounded waits, descriptors, MMAs, TMEM and TMA accesses, tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace iie {

constexpr unsigned TL_WAIT_LIMIT = 1u << 17;
constexpr int TL_SIXTEEN_FROM = 288;

__device__ __forceinline__ uint32_t tl_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tl_init(uint32_t b, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(n)); }
__device__ __forceinline__ void tl_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(b) : "memory"); }
__device__ __forceinline__ void tl_expect(uint32_t b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tl_try(uint32_t b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(b), "r"(parity) : "memory");
    return ok != 0;
}
static __device__ __noinline__ bool tl_wait_slow(uint32_t b, uint32_t parity, volatile int *abort_flag) {      // bounded
    for (unsigned it = 0; it < TL_WAIT_LIMIT; it++) {
        uint32_t ok;                                               // asleep for up to 20 us at a time
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(b), "r"(parity), "r"(20000u) : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ bool tl_wait(uint32_t b, uint32_t parity, volatile int *abort_flag) {        // the whole warp, one answer
    if (__all_sync(0xffffffffu, tl_try(b, parity))) return true;
    return __all_sync(0xffffffffu, tl_wait_slow(b, parity, abort_flag));
}
__device__ __forceinline__ uint32_t tl_elect() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
    return r;
}
// split tiles: the same shared-memory address in another CTA of the cluster, and what goes there
__device__ __forceinline__ uint32_t tl_remote(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void tl_remote_store(uint32_t a, i128 v) {
    asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"((unsigned long long)v), "l"((unsigned long long)((u128)v >> 64)) : "memory");
}
__device__ __forceinline__ void tl_remote_arrive(uint32_t b) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(b) : "memory"); }
static __device__ __noinline__ bool tl_wait_cluster(uint32_t b, uint32_t parity, volatile int *abort_flag) {       // bounded; the whole warp, one answer
    bool done = false;
    for (unsigned it = 0; it < TL_WAIT_LIMIT && !done && !*abort_flag; it++) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok) : "r"(b), "r"(parity), "r"(20000u) : "memory");
        done = ok != 0;
    }
    if (!done) *abort_flag = 1;
    return __all_sync(0xffffffffu, done);
}
__device__ __forceinline__ void tl_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// a position in a ring of slots, stepped (a division by a run-time slot count in every role's loop costs hundreds of clocks)
struct TlRing {
    int slot = 0;
    uint32_t pass = 0;
    bool lapped = false;
    __device__ __forceinline__ void step(int n) { if (++slot == n) { slot = 0; pass ^= 1; lapped = true; } }
};
// K-major operands: rows of 128 bytes with the 128-byte swizzle, rows of 32 bytes with the 32-byte swizzle
__device__ __forceinline__ uint64_t tl_desc128(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFF) | (1ULL << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ULL << 46) | (2ULL << 61);
}
__device__ __forceinline__ uint64_t tl_desc32(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFF) | (1ULL << 16) | ((uint64_t)(256 >> 4) << 32) | (1ULL << 46) | (6ULL << 61);
}
__device__ __forceinline__ uint32_t tl_idesc(int n, bool a_signed) {     // u8 / s8 x s8 -> s32, M = 128
    return (2u << 4) | (a_signed ? 1u << 7 : 0u) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void tl_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void tl_commit(uint32_t b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(b) : "memory");
}
__device__ __forceinline__ void tl_ld4(uint32_t addr, int (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tl_tma(uint32_t dst, const CUtensorMap *map, int col, int plane, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(col), "r"(plane), "r"(row), "r"(bar) : "memory");
}
__device__ __forceinline__ void tl_sts64(uint32_t a, uint32_t x, uint32_t y) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y)); }
__device__ __forceinline__ void tl_sts32(uint32_t a, uint32_t x) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x)); }

// Whether gate / up tiles of sixteen rows take a call from those of eight, counted as each would have them: the weights are expanded once per
// tile, in eight-row tiles at two thirds of the price, so that few experts with many rows each are quicker in the larger ones once they fill the
// device.  128 experts, top 8, all tokens on the same eight: 64 / 100 / 128 tokens 126 / 172 / 194 us a block by eight rows, 109 / 153 / 169 by
// sixteen; spread over all 128 experts 221 / 259 (96 tokens) / 280 against 255 / 264 / 284; 32 experts, top 4, 64 tokens on the same four 79 / 79.  (48
// tokens on the same eight, 99 / 89, stay with eight rows: the second launch would be every call's of 33 tokens and more.)
__device__ __forceinline__ bool tl_rows_of_sixteen(long long of8, long long of16) { return 2 * of8 > 3 * of16 + TL_SIXTEEN_FROM; }

// digit planes carried for `nl` digits in use
__device__ __forceinline__ int tl_planes(int nl) { return nl <= 3 ? 3 : nl <= 6 ? nl : 8; }

using TlEncode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
inline TlEncode tl_encode() {
    static TlEncode fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<TlEncode>(p);
    }();
    return fn;
}
// [rows][planes][width] bytes, boxes of `cols` columns x `planes_box` planes x `rows_box` rows
inline bool tl_map(CUtensorMap *map, const int8_t *p, long long width, long long planes, long long rows, int cols, int rows_box, CUtensorMapSwizzle swizzle, int planes_box = 1) {
    const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)planes, (cuuint64_t)rows};
    const cuuint64_t strides[2] = {(cuuint64_t)width, (cuuint64_t)(planes * width)};
    const cuuint32_t box[3] = {(cuuint32_t)cols, (cuuint32_t)planes_box, (cuuint32_t)rows_box}, estr[3] = {1, 1, 1};
    return tl_encode()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t *>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace iie
