// Exact integer RMSNorm pieces shared by the routing kernel and the whole-step decode kernel
// (arithmetic of north-mini-code/src/nmc/_bonsai/fixedpoint.py:32-72).
#pragma once
#include "common.cuh"

namespace iie {

__host__ __device__ __forceinline__ unsigned long long uabs64(int64_t v) { return v < 0 ? (0ULL - (unsigned long long)v) : (unsigned long long)v; }

// floor(sqrt(v)).  Below 2^104 the root is under 2^52, so the double estimate is within a unit or two of it and the
// residual v - r^2 (under 2^55 in size) is exact in the low 64 bits: the fix-up walks r by the residual in 64-bit words
// (the usual case: the mean square of a residual row is far below that bound); beyond it the bitwise root.
__host__ __device__ inline u128 isqrt128(u128 v) {
    if (v < ((u128)1 << 104)) {
        const double dv = (double)(unsigned long long)(v >> 64) * 18446744073709551616.0 + (double)(unsigned long long)v;
        unsigned long long r = (unsigned long long)sqrt(dv);
        long long e = (long long)((unsigned long long)v - r * r);
        while (e < 0) { r--; e += (long long)(2 * r + 1); }                       // v - (r-1)^2 = e + 2(r-1) + 1
        while (e > (long long)(2 * r)) { e -= (long long)(2 * r + 1); r++; }      // (r+1)^2 <= v  <=>  e >= 2r + 1
        return r;
    }
    u128 res = 0, bit = (u128)1 << 126;
    while (bit > v) bit >>= 2;
    while (bit != 0) {
        if (v >= res + bit) { v -= res + bit; res = (res >> 1) + bit; } else res >>= 1;
        bit >>= 2;
    }
    return res;
}

// A reciprocal for floor_div_recip: any value from a few units below floor((2^64 - 1) / den) up to it serves (the
// quotient estimate only starts lower and the correction loop takes an extra step).  In the middle range a double
// quotient minus its error bound replaces the 64-bit division.
__host__ __device__ __forceinline__ unsigned long long recip_below(unsigned long long den) {
    if (den == 0) return 0;
    if (den >= (1ULL << 13) && den < (1ULL << 60))             // 2^64/den <= 2^51: the double quotient is within 1 of it
        return (unsigned long long)(18446744073709551616.0 / (double)den) - 4;
    return 0xFFFFFFFFFFFFFFFFULL / den;
}

// high half of a 64 x 64-bit product (the host form lets tests/host_norm_check.cu run these helpers on the CPU)
__host__ __device__ __forceinline__ unsigned long long mulhi64(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (unsigned long long)(((u128)a * b) >> 64);
#endif
}

// floor(num / den) for |num| < 2^62 and 0 < den < 2^62 through a precomputed reciprocal
// inv <= floor((2^64 - 1) / den) and within a few units of it: the estimate is a few units below the quotient at most.
__host__ __device__ __forceinline__ int64_t floor_div_recip(int64_t num, unsigned long long den, unsigned long long inv) {
    const unsigned long long n = uabs64(num);
    unsigned long long q = mulhi64(n, inv), r = n - q * den;
    while (r >= den) { q++; r -= den; }
    return num >= 0 ? (int64_t)q : -(int64_t)q - (r != 0);
}

// one element of the normalised row: floor((x << fa) / rms), then (y * gain) >> fa; `bad` is set (and 0 returned)
// where the oracle's envelope checks would refuse the value
__device__ __forceinline__ int64_t norm_value(int64_t xv, unsigned long long rms, unsigned long long inv, unsigned long long gm,
                                              int64_t g, bool has_gain, int fa, bool &bad) {
    int64_t y;
    if (inv != 0 && uabs64(xv) < (1ULL << (62 - fa))) {
        // |x << fa| < 2^62 and rms < 2^62: quotient from the reciprocal inv = floor((2^64 - 1) / rms), at most 2 low
        const unsigned long long n = uabs64(xv) << fa;
        unsigned long long q = __umul64hi(n, inv), r = n - q * rms;
        while (r >= rms) { q++; r -= rms; }
        y = xv >= 0 ? (int64_t)q : -(int64_t)q - (r != 0);      // floor toward -inf
    } else {
        const i128 num = (i128)xv << fa;
        i128 q = num / (i128)rms;
        if (num < 0 && q * (i128)rms != num) q -= 1;
        if (q > (i128)INT64_MAX || q < (i128)INT64_MIN) { bad = true; return 0; }
        y = (int64_t)q;
    }
    if (has_gain) {
        // the oracle refuses a gain product that could leave int64
        if ((u128)uabs64(y) * gm > (u128)INT64_MAX) { bad = true; return 0; }
        y = (int64_t)(((i128)y * g) >> fa);
    }
    return y;
}

// sum over the warp of 64-bit and 128-bit values: pieces of 22 bits, one warp reduction each
__device__ __forceinline__ u128 warp_sum64(uint64_t v) {
    u128 sum = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) sum += (u128)__reduce_add_sync(0xffffffffu, (uint32_t)(v >> (22 * k)) & 0x3FFFFFu) << (22 * k);
    return sum;
}
__device__ __forceinline__ u128 warp_sum128(u128 v) {
    u128 sum = warp_sum64((uint64_t)v);
    if (__any_sync(0xffffffffu, (uint64_t)(v >> 64) != 0)) sum += warp_sum64((uint64_t)(v >> 64)) << 64;
    return sum;
}

// What a normalised row's values share: the root of the mean square and how the quotients floor((x << fa) / rms) are taken.
struct NormRow {
    uint64_t rms;
    int fa, sh;                    // sh: shift behind the gain (0 without one: a factor of one)
    bool refused, fast;
    int mh, ml, post;
    // Sum of squares, bit lengths of the largest |x| and |gain|, whether an |x| is beyond 2^57 (the sum may have wrapped)
    __device__ __forceinline__ NormRow(u128 ssq, int xb, int gb, bool beyond, int width, uint64_t eps, int fa_, bool has_gain) {
        fa = fa_; sh = has_gain ? fa_ : 0;
        u128 mean;
        if ((width & (width - 1)) == 0) mean = ssq >> (31 - __clz(width));
        else mean = (ssq >> 64) == 0 ? (u128)((uint64_t)ssq / (unsigned)width) : ssq / (u128)(unsigned)width;
        const u128 root = isqrt128(mean + eps);
        rms = (uint64_t)root;
        refused = beyond || root == 0 || (root >> 64) != 0;
        // The fast form: with s = 61 + l - fa (rms has l + 1 bits), floor((x << fa) / rms) = floor(x M / 2^s) for every M on the right side
        // of 2^(fa + s) / rms (above for x >= 0, below for x < 0) whose distance d from it satisfies |x| d rms < 2^s.  The double
        // quotient is within 2^10 of it, so M = quotient -+ 2^10 serves while |x| < 2^(48 - fa).  |x| < 2^xb and |gain| < 2^gb bound
        // the quotient by 2^(xb + fa - l) and the product behind the gain by 2^(xb + fa - l + gb - sh): 32-bit words hold both,
        // and four balanced digits the product.
        const int l = 63 - __clzll((long long)rms), q_bits = xb + fa - l;
        fast = !refused && l <= 31 && xb <= 31 && xb <= 48 - fa && gb <= 31 && q_bits <= 30 && q_bits + gb - sh <= 30;
        const uint64_t m = (uint64_t)(21267647932558653966460912964485513216.0 / (double)(rms << (63 - l))) - 1024;      // 2^124
        mh = (int)(m >> 31); ml = (int)(m & 0x7FFFFFFF);
        post = 30 + l - fa;
    }
    __device__ __forceinline__ int fast_value(int x, int g) const {
        const int64_t p0 = (int64_t)x * ml + (int64_t)max(x, 0) * 2048;
        const int q = (int)(((int64_t)x * mh + (p0 >> 31)) >> post);
        return (int)(((int64_t)q * g) >> sh);
    }
};
__device__ __forceinline__ uint64_t warp_max64(uint64_t v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) { const uint64_t o = __shfl_xor_sync(0xffffffffu, v, off); v = o > v ? o : v; }
    return v;
}
// largest |gain| of a row, for the values that take the general form: the whole warp
__device__ __forceinline__ uint64_t warp_gain_max(const int64_t *gain, int width) {
    uint64_t gm = 0;
    for (int k = 0; k < width; k += 32) { const int i = k + (threadIdx.x & 31); const uint64_t v = i < width ? uabs64(gain[i]) : 0; gm = v > gm ? v : gm; }
    return warp_max64(gm);
}

}  // namespace iie
