// fixstencil.cuh -- 6th-order FP64 stencils in exact integer arithmetic.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM quarter, 64
// times fewer than 32-bit integer or FP32 instructions, and the stencils are
// 736 of the ~1180 FP64 instructions of a site and stage.  Here a stencil's
// doubles are aligned to the largest exponent among them as 64-bit integers
// (56 bits below the largest value's binade: 3 bits more than FP64), summed
// exactly with the integer weights 45, -9, 1 (60 dx times the derivative) and
// 270, -27, 2 (180 dx^2 times the Laplacian, on differences from the centre
// value), and each finished sum is rounded once to FP64; the factors stay in
// the coefficients of the physics.  A derivative carries that rounding and
// the bits below 2^-55 of the largest value on its line of neighbours (of the
// whole stencil where a Laplacian comes with it), where the
// floating-point evaluation rounds every partial sum at 2^-53 and every
// weight (3/20, 1/90, 49/6 ... are no FP64 numbers) once.  Divergences and curls
// add such sums of different arrays, each aligned by itself.
//
// A value goes to an integer by bit operations (about 12), the sums are
// add/multiply pairs, a finished sum goes back by a count of leading zeros
// and shifts (about 20): some 450 integer instructions for a gradient with
// Laplacian, against 37 FP64 instructions (2368 issue slots).  A step of the
// FP64 form at 256^3 went from 144.4 to 76.1 ms (64^3: 2.41 to 1.20) with
// these stencils and the factored physics, 1046 FP64 instructions per warp and
// stage to 501, and to 60.2 (1.01) with four warps per 32 sites (stage_fp64.cu).
//
// Stencils whose largest magnitude lies outside [2^-895, 2^977] (denormals,
// infinities and NaN among them) take the floating-point evaluation, a
// stencil of zeros gives zero.
#pragma once
#include "accessors.cuh"

namespace fix {

__device__ __forceinline__ int64_t i64(uint32_t lo, uint32_t hi) { return (int64_t)(((uint64_t)hi << 32) | lo); }

// exponent field of v, in place
__device__ __forceinline__ uint32_t exp20(double v) { return (uint32_t)__double2hiint(v) & 0x7ff00000u; }

// the exponents e20 (largest of a stencil) that the integer path covers
__device__ __forceinline__ bool covered(uint32_t e20) { return e20 - (128u << 20) < (1872u << 20); }

// zeros (either sign): the arrays a run starts without, away from what feeds them
__device__ __forceinline__ bool zero_bits(double v) {
    return (((uint32_t)__double2hiint(v) << 1) | (uint32_t)__double2loint(v)) == 0u;
}
template <int N>
__device__ __forceinline__ bool zero_bits(const double (&f)[N][6]) {
    bool z = true;
#pragma unroll
    for (int ax = 0; ax < N; ++ax)
#pragma unroll
        for (int k = 0; k < 6; ++k) z = z && zero_bits(f[ax][k]);
    return z;
}

// v in units of 2^(E - 1023 - 55), rounded towards minus infinity (a
// negative value one unit lower: stencil weights sum to zero, and the unit is
// an eighth of the largest value's last place); e20p = e20 + (7 << 20)
__device__ __forceinline__ int64_t align(double v, uint32_t e20p) {
    const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
    const uint32_t s = (uint32_t)((int32_t)h >> 31);
    const uint32_t sh = (e20p - (h & 0x7ff00000u)) >> 20;  // 7 + the distance to the largest exponent
    // 1.mantissa at bits 62..10
    const uint32_t mh = ((__funnelshift_l(l, h, 10) & 0x3fffffffu) | 0x40000000u) ^ s;
    const uint32_t ml = (l << 10) ^ s;
    return i64(ml, mh) >> min(sh, 63u);
}

// V * 2^(E - 1023 - 55 + up) rounded to nearest, |V| < 2^63
__device__ __forceinline__ double to_double(int64_t V, uint32_t e20, int up) {
    const int64_t s = V >> 63;
    uint64_t u = (uint64_t)((V ^ s) - s);
    const int n = __clzll((long long)u);
    u <<= (n - 1) & 63;  // leading one at bit 62
    u += 0x200u;
    const uint32_t hi = (uint32_t)(u >> 42), lo = (uint32_t)(u >> 10);  // leading one at bit 52 of (hi, lo): adds 1 to the exponent field
    // |V| in [2^(63 - n), 2^(64 - n)): exponent E - 55 + up + 63 - n
    const uint32_t e = e20 + (uint32_t)((8 - 1 + up) - n) * (1u << 20);
    const uint32_t r = (hi + e) | ((uint32_t)(s >> 32) & 0x80000000u);
    return V == 0 ? 0.0 : __hiloint2double((int)r, (int)lo);
}

// 45 d1 - 9 d2 + d3, |d| <= 2^57
__device__ __forceinline__ int64_t weigh_grad(int64_t d1, int64_t d2, int64_t d3) { return 45 * d1 - 9 * d2 + d3; }

// the floating-point evaluation of a derivative, f = the neighbours [+1, +2, +3, -1, -2, -3]
__device__ __forceinline__ double d1(const double* f) {
    return 45.0 * (f[0] - f[3]) - 9.0 * (f[1] - f[4]) + (f[2] - f[5]);
}
__device__ __forceinline__ uint32_t largest(const double* f) {
    uint32_t e = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) e = max(e, exp20(f[d]));
    return e;
}
// The weighted sums V of N lines of neighbours, each on the line's own exponent e.
// False: a line is not covered.
template <int N>
__device__ __forceinline__ bool weighed(const double (&f)[N][6], int64_t* V, uint32_t* e) {
    bool all = true;
#pragma unroll
    for (int ax = 0; ax < N; ++ax) {
        e[ax] = largest(f[ax]);
        all = all && covered(e[ax]);
    }
    if (!all) return false;
#pragma unroll
    for (int ax = 0; ax < N; ++ax) {
        const uint32_t ep = e[ax] + (7u << 20);
        int64_t D[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) D[d] = align(f[ax][d], ep) - align(f[ax][d + 3], ep);
        V[ax] = weigh_grad(D[0], D[1], D[2]);
    }
    return true;
}

// The sum of the N terms V 2^(E - 1023 - 55), rounded once: every term is moved
// to the unit 2^-60 of the largest term.  The lines of a divergence or a curl
// are of different arrays, and one with large values and a small derivative
// must not cost the others their last bits (values aligned to the largest of
// all lines: error 3e-11 of the divergence where one array is 1 and constant, the
// others waves of 1e-6; now 1e-16).  About 70 integer instructions more than
// that: a step 0.8% at 64^3, 1.3% at 256^3, a snapshot at 128^3 2.7%.
template <int N>
__device__ __forceinline__ double sum(const int64_t* V, const uint32_t* e20) {
    uint64_t u[N];
    int64_t s[N];
    uint32_t p[N], top = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        s[k] = V[k] >> 63;
        u[k] = (uint64_t)((V[k] ^ s[k]) - s[k]);
        const int n = __clzll((long long)u[k]);
        u[k] <<= (n - 1) & 63;  // leading one at bit 62
        p[k] = V[k] == 0 ? 0u : e20[k] + (uint32_t)(63 - n) * (1u << 20);  // its exponent
        top = max(top, p[k]);
    }
    int64_t W = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const uint64_t w = u[k] >> min(((top - p[k]) >> 20) + 2u, 63u);
        W += ((int64_t)w ^ s[k]) - s[k];
    }
    return to_double(W, top - (60u << 20), 0);
}

// gradient from the lines of one array, divergence from those of three
__device__ __forceinline__ void grad(const double (&f)[3][6], double& gx, double& gy, double& gz) {
    int64_t V[3];
    uint32_t e[3];
    if (weighed(f, V, e)) {
        gx = to_double(V[0], e[0], 0);
        gy = to_double(V[1], e[1], 0);
        gz = to_double(V[2], e[2], 0);
    } else {
        const bool z = (e[0] | e[1] | e[2]) == 0u && zero_bits(f);
        gx = z ? 0.0 : d1(f[0]);
        gy = z ? 0.0 : d1(f[1]);
        gz = z ? 0.0 : d1(f[2]);
    }
}
__device__ __forceinline__ double div(const double (&f)[3][6]) {
    int64_t V[3];
    uint32_t e[3];
    if (weighed(f, V, e)) return sum<3>(V, e);
    return (e[0] | e[1] | e[2]) == 0u && zero_bits(f) ? 0.0 : d1(f[0]) + d1(f[1]) + d1(f[2]);
}

// (270 t1 - 27 t2 + 2 t3) >> 6, |t| < 2^60, without overflow
__device__ __forceinline__ int64_t weigh_lap(int64_t t1, int64_t t2, int64_t t3) {
    const int64_t lo = (int64_t)((uint64_t)(uint32_t)t1 * 270u + (uint64_t)(uint32_t)t3 * 2u) -
                       (int64_t)((uint64_t)(uint32_t)t2 * 27u);
    const int64_t hi = (int64_t)(int32_t)(t1 >> 32) * 270 + (int64_t)(int32_t)(t3 >> 32) * 2 -
                       (int64_t)(int32_t)(t2 >> 32) * 27 + (lo >> 32);
    return (hi << 26) | (int64_t)((uint32_t)lo >> 6);
}

}  // namespace fix

// FP64 stencils of the stage kernels on the integer pipes, first derivatives
// and divergences times 60 dx, Laplacians times 180 dx^2.  The neighbours'
// offsets are found from (i, j, k) for each stencil anew, some 50 integer
// instructions, instead of 18 registers that live through all of them.
struct FixAcc {
    const Ptr36& X;
    const Grid& g;
    int i, j, k, c;

    __device__ __forceinline__ const double* at(int a) const { return reinterpret_cast<const double*>(X.p[a]) + c; }
    __device__ __forceinline__ double v(int a) const { return __ldg(at(a)); }
    // plane k of the lattice, or (g.zg > 0) interior plane k of a slab
    __device__ __forceinline__ void place(int i_, int j_, int k_) {
        i = i_;
        j = j_;
        k = k_;
        c = i + g.nx * (j + g.ny * (k + g.zg));
    }
    // the neighbours [+1, +2, +3, -1, -2, -3] of *p along an axis
    __device__ __forceinline__ void along(const double* p, int ax, double* f) const {
        int q = ax == 0 ? i : (ax == 1 ? j : k);
        asm volatile("" : "+r"(q));  // keeps the offsets from being hoisted out of the caller's loop
        const int stride = ax == 0 ? 1 : (ax == 1 ? g.nx : g.nx * g.ny);
        const int n = ax == 0 ? g.nx : (ax == 1 ? g.ny : (g.zg ? 1 << 30 : g.nz));
        if (ax == 2 && g.zg) q = 1 << 29;  // ghost planes
#pragma unroll
        for (int d = 1; d <= 3; ++d) {
            f[d - 1] = __ldg(p + (q + d < n ? d : d - n) * stride);
            f[d + 2] = __ldg(p + (q >= d ? -d : n - d) * stride);
        }
    }
    __device__ __forceinline__ void grad_lap(int a, double& gx, double& gy, double& gz, double& lap) const {
        const double* p = at(a);
        double f[3][6];
        const double f0 = __ldg(p);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(p, ax, f[ax]);
        const uint32_t e = max(fix::exp20(f0), max(fix::largest(f[0]), max(fix::largest(f[1]), fix::largest(f[2]))));
        if (!fix::covered(e)) {
            if (e == 0 && fix::zero_bits(f0) && fix::zero_bits(f)) {
                gx = gy = gz = lap = 0.0;
            } else {
                gx = fix::d1(f[0]);
                gy = fix::d1(f[1]);
                gz = fix::d1(f[2]);
                double S[3];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    S[d] = f[0][d] + f[0][d + 3] + (f[1][d] + f[1][d + 3]) + (f[2][d] + f[2][d + 3]);
                lap = -1470.0 * f0 + 270.0 * S[0] - 27.0 * S[1] + 2.0 * S[2];
            }
            return;
        }
        const uint32_t ep = e + (7u << 20);
        const int64_t i0 = fix::align(f0, ep);
        int64_t T[3] = {-6 * i0, -6 * i0, -6 * i0};
        double r[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            int64_t D[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int64_t u = fix::align(f[ax][d], ep), w = fix::align(f[ax][d + 3], ep);
                D[d] = u - w;
                T[d] += u + w;
            }
            r[ax] = fix::to_double(fix::weigh_grad(D[0], D[1], D[2]), e, 0);
        }
        gx = r[0];
        gy = r[1];
        gz = r[2];
        lap = fix::to_double(fix::weigh_lap(T[0], T[1], T[2]), e, 6);
    }

    __device__ __forceinline__ void grad(int a, double& gx, double& gy, double& gz) const {
        const double* p = at(a);
        double f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(p, ax, f[ax]);
        fix::grad(f, gx, gy, gz);
    }

    // dx(a) + dy(a + 1) + dz(a + 2)
    __device__ __forceinline__ double div3(int a) const {
        double f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(at(a + ax), ax, f[ax]);
        return fix::div(f);
    }
};

// First derivatives of an FP64 [36][S] buffer for the diagnostics, 60 dx times
// their value.
struct FixDiff {
    const double* y;
    int64_t S;
    int c;
    int o[3][6];  // [+1, +2, +3, -1, -2, -3] along x, y, z

    __device__ __forceinline__ double v(int q) const { return __ldg(y + q * S + c); }
    __device__ __forceinline__ void along(int q, int ax, double* f) const {
#pragma unroll
        for (int k = 0; k < 6; ++k) f[k] = __ldg(y + q * S + c + o[ax][k]);
    }
    __device__ __noinline__ void grad(int q, double& gx, double& gy, double& gz) const {
        double f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(q, ax, f[ax]);
        fix::grad(f, gx, gy, gz);
    }
    // d_a q - d_b r
    __device__ __noinline__ double curl(int q, int a, int r, int b) const {
        double f[2][6];
        along(q, a, f[0]);
        along(r, b, f[1]);
        int64_t V[2];
        uint32_t e[2];
        if (!fix::weighed(f, V, e)) return (e[0] | e[1]) == 0u && fix::zero_bits(f) ? 0.0 : fix::d1(f[0]) - fix::d1(f[1]);
        V[1] = -V[1];
        return fix::sum<2>(V, e);
    }
    // dx q + dy (q + 1) + dz (q + 2)
    __device__ __noinline__ double div(int q) const {
        double f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(q + ax, ax, f[ax]);
        return fix::div(f);
    }
};
