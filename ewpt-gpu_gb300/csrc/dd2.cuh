// dd2.cuh -- double-float arithmetic (dd.cuh) for two lattice sites at once:
// hi and lo are packed float pairs, every operation one FADD2 / FMUL2 / FFMA2
// for both sites, half the instructions of two scalar sequences.
//
// Values stay unnormalised through sums and products: an addition is Knuth's
// TwoSum on the high parts plus the low parts (8 operations, 11 with dd's
// renormalisation), a product the FMA error of the high parts plus the cross
// terms (4, 7 with it).  Finished derivatives, currents and rates are
// renormalised (done2).  TwoSum holds whatever the order of its operands, and a
// product drops the product of the low parts alone: each low part is within a
// few 2^-24 of the values that were summed to it, so the loss is ~2^-47 of the
// factors before they cancelled, as it is for normalised pairs.  Against FP64,
// 192 runs of three lattices (bubbles, thermal states, a drive; 1 to 40 steps):
// l2 error of the worst array 0.975 (median) of the normalised one-site form's,
// at most 1.0004; largest error 0.99 (mean; single runs 0.76 to 1.16).
#pragma once
#include "dd.cuh"
#include "f32x2.cuh"

struct dd2 {
    float2 hi, lo;
    dd2() = default;
    __host__ __device__ constexpr dd2(float2 h, float2 l) : hi(h), lo(l) {}
    __host__ __device__ explicit dd2(const dd& v) : hi{v.hi, v.hi}, lo{v.lo, v.lo} {}
    __host__ __device__ explicit dd2(double d) : dd2(dd(d)) {}
    __host__ __device__ explicit dd2(float f) : hi{f, f}, lo{0.f, 0.f} {}
    __host__ __device__ explicit dd2(int i) : dd2((double)i) {}
    __host__ __device__ explicit dd2(float4 v) : hi{v.x, v.y}, lo{v.z, v.w} {}
    __host__ __device__ float4 f4() const { return make_float4(hi.x, hi.y, lo.x, lo.y); }
};

__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }

// |hi| >= |lo|: the same value with lo at most half an ulp of hi
__device__ __forceinline__ dd2 done2(const dd2& a) {
    const float2 s = __fadd2_rn(a.hi, a.lo);
    return dd2(s, sub2(a.lo, sub2(s, a.hi)));
}
__device__ __forceinline__ dd2 operator+(const dd2& a, const dd2& b) {
    const float2 s = __fadd2_rn(a.hi, b.hi);
    const float2 v = sub2(s, a.hi);
    const float2 e = __fadd2_rn(sub2(a.hi, sub2(s, v)), sub2(b.hi, v));
    return dd2(s, __fadd2_rn(e, __fadd2_rn(a.lo, b.lo)));
}
__device__ __forceinline__ dd2 operator-(const dd2& a) { return dd2(neg2(a.hi), neg2(a.lo)); }
__device__ __forceinline__ dd2 operator-(const dd2& a, const dd2& b) { return a + (-b); }
// unnormalised product
__device__ __forceinline__ dd2 mul2(const dd2& a, const dd2& b) {
    const float2 p = __fmul2_rn(a.hi, b.hi);
    float2 e = __ffma2_rn(a.hi, b.hi, neg2(p));
    e = __ffma2_rn(a.hi, b.lo, e);
    return dd2(p, __ffma2_rn(a.lo, b.hi, e));
}
__device__ __forceinline__ dd2 operator*(const dd2& a, const dd2& b) { return mul2(a, b); }
__device__ __forceinline__ dd2 operator/(const dd2& a, const dd2& b) {
    const dd x = dd(a.hi.x, a.lo.x) / dd(b.hi.x, b.lo.x), y = dd(a.hi.y, a.lo.y) / dd(b.hi.y, b.lo.y);
    return dd2(make_float2(x.hi, y.hi), make_float2(x.lo, y.lo));
}
__device__ __forceinline__ dd2& operator+=(dd2& a, const dd2& b) { return a = a + b; }
__device__ __forceinline__ dd2& operator-=(dd2& a, const dd2& b) { return a = a - b; }
