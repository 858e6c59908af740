// f32x2.cuh -- packed pair-of-float arithmetic for two lattice sites at once.
//
// sm_100-class GPUs issue FADD2/FMUL2/FFMA2: one instruction operates on a
// pair of floats.  The FP32-form stage kernel gives each thread two
// x-adjacent sites and runs the ordinary templated physics (physics.cuh) on
// this pair type, so every flux operation is one packed instruction for two
// sites.  A product is kept unevaluated (Prod) until it meets an addition, so
// `a * b + c` becomes a single FFMA2 as the scalar compiler would contract it.
#pragma once
#include <cuda_runtime.h>

// Where two products meet, one of them is rounded first: the left one, with the
// right one fused (f2, the paired kernels' own rounding), or with FIRST the
// right one, as the scalar compiler contracts the one-site kernel's sums (s2:
// two sites with the bits of one at a time; test_gpu_pairs_as_one.py).
template <bool FIRST>
struct Prod2 {
    float2 a, b;
    __device__ __forceinline__ float2 eval() const { return __fmul2_rn(a, b); }
};

template <bool FIRST>
struct Pair2 {
    static constexpr bool kFirst = FIRST;
    using Prod = Prod2<FIRST>;
    float2 v;
    __host__ __device__ __forceinline__ Pair2() {}
    __host__ __device__ __forceinline__ Pair2(float2 x) : v(x) {}
    __host__ __device__ __forceinline__ explicit Pair2(float s) : v(make_float2(s, s)) {}
    __host__ __device__ __forceinline__ explicit Pair2(double s) : v(make_float2((float)s, (float)s)) {}
    __host__ __device__ __forceinline__ explicit Pair2(int s) : v(make_float2((float)s, (float)s)) {}
    __device__ __forceinline__ Pair2(const Prod& p) : v(p.eval()) {}
    __device__ __forceinline__ Pair2& operator+=(const Pair2& b) { return *this = *this + b; }
    __device__ __forceinline__ Pair2& operator-=(const Pair2& b) { return *this = *this - b; }
    __device__ __forceinline__ Pair2& operator+=(const Prod& b) { return *this = *this + b; }
    __device__ __forceinline__ Pair2& operator-=(const Prod& b) { return *this = *this - b; }
};
using f2 = Pair2<false>;
using s2 = Pair2<true>;

__device__ __forceinline__ float2 neg2(float2 x) { return make_float2(-x.x, -x.y); }

#define PAIR2_OP template <bool F> __device__ __forceinline__

// products
PAIR2_OP Prod2<F> operator*(const Pair2<F>& a, const Pair2<F>& b) { return {a.v, b.v}; }
PAIR2_OP Prod2<F> operator*(const Prod2<F>& a, const Pair2<F>& b) { return {a.eval(), b.v}; }
PAIR2_OP Prod2<F> operator*(const Pair2<F>& a, const Prod2<F>& b) { return {a.v, b.eval()}; }
PAIR2_OP Prod2<F> operator*(const Prod2<F>& a, const Prod2<F>& b) { return {a.eval(), b.eval()}; }
PAIR2_OP Prod2<F> operator-(const Prod2<F>& p) { return {neg2(p.a), p.b}; }

// sums
PAIR2_OP Pair2<F> operator+(const Pair2<F>& a, const Pair2<F>& b) { return __fadd2_rn(a.v, b.v); }
PAIR2_OP Pair2<F> operator-(const Pair2<F>& a, const Pair2<F>& b) { return __fadd2_rn(a.v, neg2(b.v)); }
PAIR2_OP Pair2<F> operator-(const Pair2<F>& a) { return neg2(a.v); }
PAIR2_OP Pair2<F> operator+(const Pair2<F>& x, const Prod2<F>& p) { return __ffma2_rn(p.a, p.b, x.v); }
PAIR2_OP Pair2<F> operator+(const Prod2<F>& p, const Pair2<F>& x) { return __ffma2_rn(p.a, p.b, x.v); }
PAIR2_OP Pair2<F> operator-(const Pair2<F>& x, const Prod2<F>& p) { return __ffma2_rn(neg2(p.a), p.b, x.v); }
PAIR2_OP Pair2<F> operator-(const Prod2<F>& p, const Pair2<F>& x) { return __ffma2_rn(p.a, p.b, neg2(x.v)); }
PAIR2_OP Pair2<F> operator+(const Prod2<F>& p, const Prod2<F>& q) {
    return F ? __ffma2_rn(p.a, p.b, q.eval()) : __ffma2_rn(q.a, q.b, p.eval());
}
PAIR2_OP Pair2<F> operator-(const Prod2<F>& p, const Prod2<F>& q) {
    return F ? __ffma2_rn(p.a, p.b, neg2(q.eval())) : __ffma2_rn(neg2(q.a), q.b, p.eval());
}

// one division per site in the physics (1/|Phi|^2): two scalar divides
PAIR2_OP Pair2<F> operator/(const Pair2<F>& a, const Pair2<F>& b) {
    return make_float2(a.v.x / b.v.x, a.v.y / b.v.y);
}
PAIR2_OP Pair2<F> operator/(const Pair2<F>& a, const Prod2<F>& b) { return a / Pair2<F>(b); }
#undef PAIR2_OP

// Error-free transformations on packed pairs (Knuth's TwoSum; the product
// error by one fused multiply-add), for the compensated stencils of the
// FP32 form's compensated mode (accessors.cuh PairAcc::grad_lap_c).
// s + e == a + b exactly (s or e may be the object a or b refers to)
__device__ __forceinline__ void two_sum2(const f2& a, const f2& b, f2& s, f2& e) {
    const f2 x = a, y = b;
    const f2 r = x + y;
    const f2 bb = r - x;
    e = (x - (r - bb)) + (y - bb);
    s = r;
}
// p + e == a * b exactly (p or e may be the object a or b refers to)
__device__ __forceinline__ void two_prod2(const f2& a, const f2& b, f2& p, f2& e) {
    const f2 x = a, y = b;
    const f2 r = f2(x * y);
    e = x * y - r;
    p = r;
}
