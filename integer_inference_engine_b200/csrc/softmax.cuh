// The two scalar steps of the fixed-point softmax where fa <= 23 (arithmetic: attn.cu), shared by the attention kernels.
#pragma once
#include "common.cuh"

namespace iie {

// exp2_neg_fixed of (d log2e) >> fa for 0 <= d <= clip: every operand fits 32 bits
struct SoftmaxExp {
    uint32_t c0 = 65536, c1 = 45426, c2 = 15743, c3 = 3638, log2e;
    int fa;
    long long clip;
    __device__ __forceinline__ SoftmaxExp(int fa_, long long log2e_, long long clip_) : log2e((uint32_t)log2e_), fa(fa_), clip(clip_) {
        const int s = 16 - fa;
        if (s >= 0) { c0 >>= s; c1 >>= s; c2 >>= s; c3 >>= s; } else { c0 <<= -s; c1 <<= -s; c2 <<= -s; c3 <<= -s; }
    }
    __device__ __forceinline__ uint32_t mul(uint32_t x, uint32_t y) const { return (uint32_t)(((uint64_t)x * y) >> fa); }
    // distance of a score below the row's maximum (not negative)
    __device__ __forceinline__ int operator()(long long below) const {
        const uint32_t u = mul((uint32_t)min(below, clip), log2e), f = u & ((1u << fa) - 1), f2 = mul(f, f), f3 = mul(f2, f);
        const int p = (int)(c0 - mul(c1, f) + mul(c2, f2) - mul(c3, f3));
        return max(p, 0) >> (u >> fa);
    }
};

// floor((e << fa) / z) for 0 <= e <= 2^fa <= z: with z of l + 1 bits and s = 61 + l - fa it is e M >> s for every M from 2^(fa + s) / z up to
// 2^11 more (e 2^11 z < 2^s); the double quotient is within 2^10.  z = 0 gives 0.
struct SoftmaxQuotient {
    uint32_t mh = 0, ml = 0;
    int post = 0;
    __device__ __forceinline__ SoftmaxQuotient(unsigned long long z, int fa) {
        if (z == 0) return;
        const int l = 63 - __clzll((long long)z);
        const uint64_t m = (uint64_t)(21267647932558653966460912964485513216.0 / (double)(z << (63 - l))) + 1024;      // 2^124
        mh = (uint32_t)(m >> 31); ml = (uint32_t)(m & 0x7FFFFFFF);
        post = 30 + l - fa;
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t e) const { return (uint32_t)(((uint64_t)e * mh + (((uint64_t)e * ml) >> 31)) >> post); }
};

}  // namespace iie
