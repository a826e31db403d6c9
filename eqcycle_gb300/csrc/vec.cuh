// Four-wide vector access for the HBM-bound vector kernels: one 16-byte access per four
// floats, two per four doubles.  Every node vector of the library starts on a 32-byte
// boundary (cudaMalloc alignment plus a row pitch that is a multiple of 8 entries), so
// interior slices [ld, size) are 16-byte aligned as well.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace eqc {

// One wave of CTAs of 256 threads, four per SM of a GB300 for FP32 vectors, three for FP64 ones, fewer where n
// has fewer 4-wide chunks.  More threads have more loads in flight, fewer pay less for the ends of their sums:
// ms per quasi-static step with two CTAs per SM, with four and three, and with six and four, 480 x 960 elements 7.59,
// 7.43 and 7.42, 240 x 480 2.68, 2.66 and 2.66, 120 x 240 1.524, 1.517 and 1.517, plain FP64 the same.
constexpr int VEC_THREADS = 256;
template <class T> constexpr int VEC_PER_SM = sizeof(T) == 4 ? 4 : 3;
template <class T> inline int vec_blocks(int64_t n) {
    const int64_t b = (n / 4 + VEC_THREADS - 1) / VEC_THREADS, most = 152 * VEC_PER_SM<T>;
    return (int)(b < 1 ? 1 : (b < most ? b : most));
}

__device__ __forceinline__ void ld4(const float* p, float (&a)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&a)[4]) {
    const double2 u = reinterpret_cast<const double2*>(p)[0], w = reinterpret_cast<const double2*>(p)[1];
    a[0] = u.x; a[1] = u.y; a[2] = w.x; a[3] = w.y;
}
__device__ __forceinline__ void st4(float* p, const float (&a)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&a)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a[0], a[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(a[2], a[3]);
}

// FP32 -> FP64, exact, by integer operations on the bit patterns (GB300 converts to FP64 on its
// FP64 unit, a small fraction of its integer and FP32 rate).  Zeros, subnormals, infinities
// and NaNs included.
__device__ __forceinline__ double f32_to_f64(float f) {
    const uint32_t b = __float_as_uint(f);
    const uint64_t sign = (uint64_t)(b >> 31) << 63;
    const uint32_t e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
    if (e == 0xffu) return __longlong_as_double((long long)(sign | (0x7ffull << 52) | ((uint64_t)m << 29)));
    if (e != 0) return __longlong_as_double((long long)(sign | ((uint64_t)(e + 896u) << 52) | ((uint64_t)m << 29)));
    if (m == 0) return __longlong_as_double((long long)sign);
    const int p = 31 - __clz((int)m);                 // leading one of a subnormal: m * 2^-149
    const uint64_t frac = ((uint64_t)m - (1ull << p)) << (52 - p);
    return __longlong_as_double((long long)(sign | ((uint64_t)(p + 874) << 52) | frac));
}

// Dot-product accumulator.  FP64 vectors accumulate in FP64.  FP32 vectors accumulate the
// exact products (a*b = p + e, e by FMA) in an unevaluated FP32 pair (hi + lo, Knuth's
// TwoSum), about 44 significant bits, then hand a double to the cross-thread reduction (reduce.cuh):
// FP64-class dot products of FP32 vectors without FP64 arithmetic per element (GB300's FP64
// and FP32<->FP64 conversion rates are a small fraction of its FP32 rate).
template <class T> struct DotAcc;
template <> struct DotAcc<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double a, double b) { s = fma(a, b, s); }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct DotAcc<float> {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float a, float b) {
        const float p = __fmul_rn(a, b);
        const float e = __fmaf_rn(a, b, -p);
        const float s = __fadd_rn(hi, p);
        const float bb = __fsub_rn(s, hi);
        const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(err, e));
    }
    __device__ __forceinline__ double value() const { return f32_to_f64(hi) + f32_to_f64(lo); }
};

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace eqc
