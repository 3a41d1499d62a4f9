// What the search kernels share: the reference's scan, the margin of the filter in front of it (derived in
// ccs_argmin.cu) and the selection of the keys within that margin.
#pragma once
#include <cstdint>

namespace lutamm {

constexpr float kEps = 1e-6f;  // (double)diff > 1e-6  <=>  diff > 1e-6f for fp32 diff
constexpr float kHuge = 1e30f;  // beyond this the filter's own arithmetic could overflow

__host__ __device__ constexpr float margin_factor(int v) { return (float)(8 * v + 16) * 5.9604644775390625e-08f; }
constexpr float kMarginBase = 0.51e-6f;

__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// smallest of n values, as a tree of three-input minima
template <int N>
__device__ __forceinline__ float min_of(const float (&k)[N]) {
    if constexpr (N == 1) {
        return k[0];
    } else if constexpr (N == 2) {
        return fminf(k[0], k[1]);
    } else {
        float t[(N + 2) / 3];
#pragma unroll
        for (int i = 0; i < N / 3; ++i) t[i] = min3(k[3 * i], k[3 * i + 1], k[3 * i + 2]);
        if constexpr (N % 3 == 1) t[N / 3] = k[N - 1];
        if constexpr (N % 3 == 2) t[N / 3] = fminf(k[N - 2], k[N - 1]);
        return min_of(t);
    }
}

// One bit per key that lies below the threshold: key i at bit i.  The comparison is the sign of key - threshold;
// NaN and overflow are excluded by the callers' check of the margin.  (Two scalar multiply-adds per key, the first
// saturating to 0 or 1, need no integer instruction but measured 4 % slower: a scalar multiply-add holds its pipe
// as long as a packed one.)
template <int N>
__device__ __forceinline__ uint32_t below(const float (&k)[N], float thr) {
    uint32_t mask = 0;
    const float2 neg = make_float2(-thr, -thr);
#pragma unroll
    for (int i = N - 2; i >= 0; i -= 2) {
        const float2 e = __fadd2_rn(make_float2(k[i], k[i + 1]), neg);
        mask = __funnelshift_l(__float_as_uint(e.y), mask, 1);
        mask = __funnelshift_l(__float_as_uint(e.x), mask, 1);
    }
    return mask;
}
// position of the highest set bit
__device__ __forceinline__ uint32_t high_bit(uint32_t v) {
    uint32_t r;
    asm("bfind.u32 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t all_but_lowest(uint32_t mask) { return mask & (mask - 1); }

// The reference's scan.  cent(c, d) returns the NEGATED component, so x - c is x + (-c): the same IEEE result.
template <int V, typename F>
__device__ __forceinline__ uint32_t exact_scan(const float (&x)[V], uint32_t CT, F cent) {
    float mn = 0.f;
    uint32_t best = 0;
#pragma unroll 1
    for (uint32_t c = 0; c < CT; ++c) {
        float acc = 0.f;
#pragma unroll
        for (int d = 0; d < V; ++d) {
            const float e = __fadd_rn(x[d], cent(c, d));
            acc = __fadd_rn(acc, __fmul_rn(e, e));
        }
        const bool take = c == 0 || __fsub_rn(mn, acc) > kEps;  // false for NaN: keeps the earlier index
        mn = take ? acc : mn;
        best = take ? c : best;
    }
    return best;
}

}  // namespace lutamm
