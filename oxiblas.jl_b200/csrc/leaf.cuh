// Pivot search of the panel leaves (real and complex): warp-wide arg-max.
#pragma once
#include <climits>
#include <cstdint>

namespace oxi {

// ---------------------------------------------------------------------------
// Warp arg-max for the pivot search with redux.sync: |v| >= 0 orders like its
// bit pattern, so the warp maximum is an integer max (FP64: high word, then
// low word), and the first row among equal maxima is an integer min of the
// positions -- the reference's "largest |a|, first row on ties".  NaN maps to
// the smallest key, as a NaN never wins the reference's strict '>' comparison.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t redux_max_u32(uint32_t v) {
    uint32_t r;
    asm volatile("redux.sync.max.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t redux_min_u32(uint32_t v) {
    uint32_t r;
    asm volatile("redux.sync.min.u32 %0, %1, 0xffffffff;" : "=r"(r) : "r"(v));
    return r;
}
// (integer instructions only: an FP64 compare or absolute value takes the FP64 pipe)
__device__ __forceinline__ bool is_nan(float a) { return (__float_as_uint(a) << 1) > 0xff000000u; }
__device__ __forceinline__ bool is_nan(double a) {
    const uint64_t b = (uint64_t)__double_as_longlong(a) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull;
}
__device__ __forceinline__ bool is_zero(float a) { return (__float_as_uint(a) << 1) == 0u; }
__device__ __forceinline__ bool is_zero(double a) {
    return ((((uint32_t)__double2hiint(a)) << 1) | (uint32_t)__double2loint(a)) == 0u;
}
__device__ __forceinline__ uint64_t pivot_key(float a) { return (uint64_t)(__float_as_uint(a) & 0x7fffffffu); }
__device__ __forceinline__ uint64_t pivot_key(double a) {
    return (uint64_t)__double_as_longlong(a) & 0x7fffffffffffffffull;
}
// The key of value a at position pos in step j: a NaN at position j keeps row j
// (the largest key), a NaN below never wins (key 0).
template <typename T>
__device__ __forceinline__ uint64_t step_key(T a, int pos, int j) {
    return is_nan(a) ? (pos == j ? ~0ull : 0ull) : pivot_key(a);
}
// The winner's lane as a one-bit mask, the same in every lane (0: no lane has a
// candidate; pos = INT_MAX marks a lane without one).  A single largest high
// word, the usual case, ends it after one reduction.
template <typename T>
__device__ __forceinline__ uint32_t warp_winner(uint64_t key, int pos) {
    const bool has = pos != INT_MAX;
    uint32_t m;
    if constexpr (sizeof(T) == 4) {
        const uint32_t k = (uint32_t)key;
        const uint32_t mk = redux_max_u32(has ? k : 0u);
        m = __ballot_sync(0xffffffffu, has && k == mk);
    } else {
        const uint32_t hi = (uint32_t)(key >> 32), lo = (uint32_t)key;
        const uint32_t mh = redux_max_u32(has ? hi : 0u);
        bool in = has && hi == mh;
        m = __ballot_sync(0xffffffffu, in);
        if (m & (m - 1)) {
            const uint32_t ml = redux_max_u32(in ? lo : 0u);
            m = __ballot_sync(0xffffffffu, in && lo == ml);
        }
    }
    if (m & (m - 1)) {
        const bool in = (m >> (threadIdx.x & 31)) & 1;
        const uint32_t mp = redux_min_u32(in ? (uint32_t)pos : (uint32_t)INT_MAX);
        m = __ballot_sync(0xffffffffu, in && (uint32_t)pos == mp);
    }
    return m;
}

// N elements between registers and 16-byte-aligned shared memory.
template <typename T, int N>
__device__ __forceinline__ void store_row(T *dst, const T *v) {
    constexpr int VEC = 16 / sizeof(T);
#pragma unroll
    for (int c = 0; c < N; c += VEC) {
        int4 x;
        T *xx = (T *)&x;
#pragma unroll
        for (int e = 0; e < VEC; ++e) xx[e] = v[c + e];
        *(int4 *)(dst + c) = x;
    }
}
template <typename T, int N>
__device__ __forceinline__ void load_row(T *v, const T *src) {
    constexpr int VEC = 16 / sizeof(T);
#pragma unroll
    for (int c = 0; c < N; c += VEC) {
        const int4 x = *(const int4 *)(src + c);
        const T *xx = (const T *)&x;
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[c + e] = xx[e];
    }
}

}  // namespace oxi
