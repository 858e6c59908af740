// host_device.h -- the device functions that the library's per-site code calls,
// for a host C++ compiler (test infrastructure, never linked into libewpt).
#pragma once
#define EWPT_ARITH inline
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef __noinline__
#define __noinline__ __attribute__((noinline))
#endif

using std::max;
using std::min;

template <typename T>
inline T __ldg(const T* p) {
    return *p;
}
inline uint64_t bits_of(double v) {
    uint64_t b;
    std::memcpy(&b, &v, 8);
    return b;
}
inline int __double2hiint(double v) { return (int)(bits_of(v) >> 32); }
inline int __double2loint(double v) { return (int)(uint32_t)bits_of(v); }
inline double __longlong_as_double(long long b) {
    double v;
    std::memcpy(&v, &b, 8);
    return v;
}
inline double __hiloint2double(int hi, int lo) {
    return __longlong_as_double((long long)((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo));
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
    return (uint32_t)(((uint64_t)hi << 32 | lo) >> (32 - (n & 31)));
}
inline int __clzll(long long v) { return v == 0 ? 64 : __builtin_clzll((unsigned long long)v); }

// packed pairs: two scalar operations
inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) {
    return make_float2(std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y));
}

inline dim3 blockIdx, blockDim, threadIdx;
