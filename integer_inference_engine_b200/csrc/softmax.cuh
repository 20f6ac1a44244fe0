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

// The same two where fa <= 16, in fewer and narrower multiplications (a 32-bit product is half the price of a 64-bit one).
// Every operand of the polynomial is at most 2^16 and none of its products both factors, so that they fit 32 bits.
struct SoftmaxExp16 {
    uint32_t c0, c1, c2, c3, log2e, clip;
    int fa;
    __device__ __forceinline__ SoftmaxExp16(int fa_, long long log2e_, long long clip_)
        : c0(65536u >> (16 - fa_)), c1(45426u >> (16 - fa_)), c2(15743u >> (16 - fa_)), c3(3638u >> (16 - fa_)), log2e((uint32_t)log2e_), clip((uint32_t)clip_), fa(fa_) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t below) const {
        const uint32_t u = (uint32_t)(((uint64_t)min(below, clip) * log2e) >> fa), f = u & ((1u << fa) - 1), f2 = (f * f) >> fa, f3 = (f2 * f) >> fa;
        const int p = (int)(c0 - ((c1 * f) >> fa) + ((c2 * f2) >> fa) - ((c3 * f3) >> fa));
        return (uint32_t)(max(p, 0) >> (u >> fa));
    }
};
// For 2^l < z <= 2^(l + 1) <= 2^31, M = floor(2^(33 + l) / z) + 1 lies in (2^32, 2^33) and floor((e << fa) / z) = (e M) >> (33 + l - fa) for
// e <= 2^fa <= z: with d = M z - 2^(33 + l) <= z the right side's quotient is e d / (z 2^(33 + l - fa)) above the left one's, less than 1 / z
// (or 1 / z with e = 2^fa and z a power of two, where the quotient is whole).  e = 0 for every key where z = 0.
struct SoftmaxQuotient16 {
    uint32_t m = 0;                                                // M - 2^32
    int post = 0;
    __device__ __forceinline__ SoftmaxQuotient16(unsigned long long z, int fa) {
        if (z == 0) return;
        const int l = 63 - __clzll((long long)(z - 1));
        const unsigned long long n = 1ULL << (33 + l);
        unsigned long long q = (unsigned long long)((double)n / (double)z);
        long long r = (long long)(n - q * z);
        while (r < 0) { q--; r += (long long)z; }
        while (r >= (long long)z) { q++; r -= (long long)z; }
        m = (uint32_t)(q + 1);
        post = 1 + l - fa;
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t e) const { return (__umulhi(e, m) + e) >> post; }
};

}  // namespace iie
