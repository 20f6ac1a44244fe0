// silu_up_fixed and silu_up_any (csrc/common.cuh) compiled for the CPU; tests/test_silu_up_cpu.py compares it with the NumPy checker.
#include "common.cuh"

extern "C" void h_silu_up(const int64_t *g, const int64_t *u, int64_t *y, long long n, int fa) {
    for (long long i = 0; i < n; i++) y[i] = iie::silu_up_fixed(g[i], u[i], fa, iie::sigmoid_log2e(fa), iie::sigmoid_clip(fa));
}
extern "C" void h_silu_up_any(const int64_t *g, const int64_t *u, int64_t *y, long long n, int fa) {
    for (long long i = 0; i < n; i++) y[i] = iie::silu_up_any(g[i], u[i], fa, iie::sigmoid_log2e(fa), iie::sigmoid_clip(fa));
}
