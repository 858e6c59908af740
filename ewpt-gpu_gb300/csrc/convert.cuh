// convert.cuh -- FP64 <-> float-pair conversions of the state arrays.
//
// A state of the FP32 form (hi, lo) and of the DF64 form is the pair
//   hi = fl32(v), lo = fl32(v - hi);   v = hi + lo rounded to FP64.
// Written with C casts, a value costs four (split) or three (join)
// instructions of the FP64 pipe, which on GB300 takes one warp instruction
// per 16 cycles and SM: at 256^3 (604 M values) that alone is 3.8 / 2.9 ms,
// against 1.4 ms for the memory traffic.  Here the split is integer
// arithmetic on the bits plus one int-to-float conversion, and the join keeps
// the one FP64 addition that rounds; both give the casts' results bit for
// bit and take the casts outside the exponent range they cover.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// hi = fl32(v), lo = fl32(v - hi)
__device__ __forceinline__ void split_f64(double v, float& hi, float& lo) {
    const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
    const uint32_t e = (h >> 20) & 0x7ff, sign = h & 0x80000000u;
    if (e - 949u <= 200u) {
        // 2^-74 <= |v| < 2^127: hi is a normal float, and lo (a multiple of
        // 2^(e - 1075) >= 2^-126) is zero or one too
        const uint32_t r = l & 0x1fffffffu;  // the 29 bits below hi's last
        const uint32_t t = (sign | ((e - 896u) << 23)) | ((h & 0xfffffu) << 3) | (l >> 29);
        const uint32_t up = (r + (t & 1u)) > 0x10000000u;  // round to nearest, ties to even
        hi = __uint_as_float(t + up);  // a carry into the exponent is the next binade (or infinity)
        int32_t q = (int32_t)r - (int32_t)(up << 29);
        q = sign ? -q : q;
        lo = (float)q * __uint_as_float((e - 948u) << 23);  // times 2^(e - 1075): exact
    } else if (((h << 1) | l) == 0u) {
        hi = __uint_as_float(h);
        lo = 0.f;
    } else {
        hi = (float)v;
        lo = (float)(v - (double)hi);
    }
}

// the double of a float (every float is one)
__device__ __forceinline__ double widen_f32(float f) {
    const uint32_t b = __float_as_uint(f);
    const uint32_t m = b & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u)  // normal
        return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + (896u << 20))), (int)(b << 29));
    if (m == 0u) return __hiloint2double((int)b, 0);
    return (double)f;
}

__device__ __forceinline__ double join_f64(float hi, float lo) { return widen_f32(hi) + widen_f32(lo); }
