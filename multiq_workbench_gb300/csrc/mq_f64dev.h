// Device helpers of the FP64 step kernels (mq_f64.cu, mq_tandem.cu): what keeps comparisons, conversions
// and the collision test off GB300's FP64 pipe, with the same results. Include from units compiled
// without FMA contraction.
#pragma once
#include "mq_phys.h"

namespace mqf {

constexpr unsigned FULL = 0xffffffffu;

// Comparisons and integer <-> double conversions of the step on the integer pipe. GB300's FP64 pipe
// limits this kernel and also executes FP64 compares and conversions; these helpers give the same
// results from the doubles' bit patterns (IEEE doubles of one sign order like their bits as
// integers), NaN and signed zeros included.
__device__ __forceinline__ bool is_nan_bits(long long b) { return (b & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL; }
// x > c for a constant c > 0
__device__ __forceinline__ bool gt_pos(long long x, long long c) { return x > c && x <= 0x7FF0000000000000LL; }
// x < c for a constant c > 0 (negative numbers and -0 included, NaN excluded)
__device__ __forceinline__ bool lt_pos(long long x, long long c) { return x < c && !is_nan_bits(x); }
// x < 0
__device__ __forceinline__ bool lt_zero(long long x) { return x < 0 && x != (long long)0x8000000000000000ULL && !is_nan_bits(x); }
// (g.max(0.0) as usize).min(n - 2) from the bits of g; lim = the bits of (double)(n - 2)
__device__ __forceinline__ int32_t cell_lo_bits(double g, int32_t n, long long lim) {
    const long long b = __double_as_longlong(g);
    if (b <= 0 || b > 0x7FF0000000000000LL) return 0;   // !(g > 0): zeros, negatives, NaN
    if (b >= lim) return n - 2;                          // g >= n - 2, +inf included
    const int e = (int)(b >> 52) - 1023;                 // 0 < g < n - 2 < 2^31
    if (e < 0) return 0;
    return (int32_t)(((b & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL) >> (52 - e));
}
// (double)v for 0 <= v < 2^31, exactly
__device__ __forceinline__ double i2d_bits(int32_t v) {
    if (v == 0) return 0.0;
    const int e = 31 - __clz(v);
    const unsigned long long m = ((unsigned long long)(uint32_t)v << (52 - e)) & 0xFFFFFFFFFFFFFULL;
    return __longlong_as_double((long long)(((unsigned long long)(1023 + e) << 52) | m));
}

// 0.0 + p, on the integer pipe: p itself, but +0 for -0
__device__ __forceinline__ double plus_zero(double p) {
    return __double_as_longlong(p) == (long long)0x8000000000000000ULL ? 0.0 : p;
}
__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(FULL, v, src); }
// order-preserving signed key of a double's bits (NaN aside; -0 as +0)
__device__ __forceinline__ long long order_key(long long b) {
    if (b == (long long)0x8000000000000000ULL) b = 0;
    return b < 0 ? (long long)(0x8000000000000000ULL - (unsigned long long)b) : b;
}
// x > c, c given by its key
__device__ __forceinline__ bool gt_key(long long x, long long key) { return !is_nan_bits(x) && order_key(x) > key; }
// FP32 upper bound of |v| from the high word of a double; from 2^127 on (infinities and NaN too) a
// value whose square overflows
__device__ __forceinline__ float mag_up(double v) {
    const int hi = min(max(__double2hiint(v) & 0x7fffffff, 0x38100000), 0x47e00000);
    return __int_as_float(((hi - 0x38000000) << 3) + 8);
}
__device__ __forceinline__ uint64_t xs_step(uint64_t x) {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return x;
}
__device__ __forceinline__ double xs_unit(uint64_t x) { return (double)(x >> 11) / 9007199254740992.0; }

}  // namespace mqf
