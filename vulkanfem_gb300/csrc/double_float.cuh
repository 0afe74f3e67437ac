// double_float.cuh -- "df" numbers: the unevaluated sum hi + lo of two FP32 values,
// about 48 significant bits, computed with FP32 instructions only (Dekker 1971:
// TwoSum / FastTwoSum; the product error from one FMA).  GB300 issues FP64 at about
// 1/64 of its FP32 rate, so the mixed-precision solve evaluates its true residual
// f - K x in df where the FP64 product is not in fixed point: relative rounding
// ~1e-14 of the summed magnitudes, 3 times faster than the FP64 march (dense Ke 1.4).  Addition is
// the "sloppy" variant (error bounded by ~2^-44 (|a| + |b|)), ample for a residual
// that is compared with 1e-6 |f|.  The compiler must not re-associate these
// expressions, which nvcc does not do without fast-math flags.
#pragma once

namespace vfem {
namespace {

struct df {
    float hi, lo;
    df() = default;
    __host__ __device__ constexpr df(float h, float l) : hi(h), lo(l) {}
    __host__ __device__ constexpr explicit df(int v) : hi((float)v), lo(0.f) {}
    __host__ __device__ constexpr explicit df(float v) : hi(v), lo(0.f) {}
    __host__ __device__ explicit df(double v) : hi((float)v), lo((float)(v - (double)(float)v)) {}
};

__device__ __forceinline__ df dfTwoSum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return df(s, (a - (s - bb)) + (b - bb));
}
__device__ __forceinline__ df dfFastTwoSum(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return df(s, b - (s - a));
}
__device__ __forceinline__ df operator+(df a, df b) {
    const df s = dfTwoSum(a.hi, b.hi);
    return dfFastTwoSum(s.hi, s.lo + (a.lo + b.lo));
}
__device__ __forceinline__ df operator-(df a, df b) { return a + df(-b.hi, -b.lo); }
__device__ __forceinline__ df operator*(df a, df b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, e);
    e = fmaf(a.lo, b.hi, e);
    return dfFastTwoSum(p, e);
}
__device__ __forceinline__ df& operator+=(df& a, df b) { return a = a + b; }
__device__ __forceinline__ df& operator*=(df& a, df b) { return a = a * b; }
// a * b + c with one renormalisation.
__device__ __forceinline__ df fma(df a, df b, df c) {
    const float p = a.hi * b.hi;
    const float pe = fmaf(a.hi, b.hi, -p);
    const df s = dfTwoSum(p, c.hi);
    float t = s.lo + (pe + c.lo);
    t = fmaf(a.hi, b.lo, t);
    t = fmaf(a.lo, b.hi, t);
    return dfFastTwoSum(s.hi, t);
}

}  // namespace
}  // namespace vfem
