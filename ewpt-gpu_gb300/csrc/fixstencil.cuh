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
// the coefficients of the physics.  A value that is aligned loses less than one
// unit, 2^-55 of the largest value on its line of neighbours (of the whole
// stencil where a Laplacian comes with it): at most 55 units in a derivative and
// 1794 in a Laplacian by the weights, and 63/64 of 64 more where the Laplacian's
// sum is cut to 64 bits.  The floating-point evaluation rounds every partial sum
// at 2^-53 and every weight (3/20, 1/90, 49/6 ... are no FP64 numbers) once.
// Divergences and curls add such sums of different arrays, each aligned by itself.
//
// A value goes to an integer by bit operations (about 12), the sums are
// add/multiply pairs, a finished sum goes back by a count of leading zeros
// and shifts (about 20): some 450 integer instructions for a gradient with
// Laplacian, against 37 FP64 instructions (2368 issue slots).  A step of the
// FP64 form at 256^3 went from 144.4 to 76.1 ms (64^3: 2.41 to 1.20) with
// these stencils and the factored physics, 1046 FP64 instructions per warp and
// stage to 501, and to 60.2 (1.01) with four warps per 32 sites (stage_fp64.cu).
//
// Every stencil of -v is minus the stencil of v to the bit, as IEEE sums are, and
// does not see the signs of zeros: a start that is symmetric under Phi -> -Phi
// or a reflection stays so.  Step times with all of this: 64^3 1.04 ms, 128^3
// 7.83, 256^3 62.0, 3% above those of sums rounded downwards on one exponent.  Values
// with exact zeros among them cost more: 64^3 1.38 ms where every array but one is
// odd in x (2.37 with floating-point stencils).
//
// Stencils whose largest magnitude lies outside [2^-895, 2^977] (denormals,
// infinities and NaN among them) take the floating-point evaluation, as do
// gradients and divergences with a zero among their values; a stencil of zeros
// gives zero.
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

// v in units of 2^(E - 1023 - 55).  Rounded towards minus infinity where no value
// of a stencil is zero: align(-v) = -align(v) - 1, and the weights sum to zero, so
// a stencil of -v is minus that of v to the bit.  A zero has no such image, and
// its sign is not to matter: NEAREST, ties away from zero, takes four
// instructions more.
template <bool NEAREST = false>
__device__ __forceinline__ int64_t align(double v, uint32_t e20) {
    const uint32_t h = (uint32_t)__double2hiint(v), l = (uint32_t)__double2loint(v);
    const uint32_t s = (uint32_t)((int32_t)h >> 31);
    const uint32_t sh = (e20 + ((NEAREST ? 6u : 7u) << 20) - (h & 0x7ff00000u)) >> 20;  // and the distance to the largest exponent
    // 1.mantissa at bits 62..10, the one's complement of a negative value's
    const uint32_t mh = ((__funnelshift_l(l, h, 10) & 0x3fffffffu) | 0x40000000u) ^ s;
    const uint32_t ml = (l << 10) ^ s;
    const int64_t q = i64(ml, mh) >> min(sh, 63u);
    return NEAREST ? (q + 1) >> 1 : q;  // q half units, or -q - 1
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
// the largest of the values' exponents; lo: down to the smallest
__device__ __forceinline__ uint32_t largest(const double* f, uint32_t& lo) {
    uint32_t e = 0;
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        e = max(e, exp20(f[d]));
        lo = min(lo, exp20(f[d]));
    }
    return e;
}
// The weighted sums V of N lines of neighbours, each on the line's own exponent e.
// False: a line is not covered or holds a zero.
template <int N>
__device__ __forceinline__ bool weighed(const double (&f)[N][6], int64_t* V, uint32_t* e) {
    uint32_t lo = ~0u;
#pragma unroll
    for (int ax = 0; ax < N; ++ax) e[ax] = largest(f[ax], lo);
    bool all = lo != 0u;
#pragma unroll
    for (int ax = 0; ax < N; ++ax) all = all && covered(e[ax]);
    if (!all) return false;
#pragma unroll
    for (int ax = 0; ax < N; ++ax) {
        int64_t D[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) D[d] = align(f[ax][d], e[ax]) - align(f[ax][d + 3], e[ax]);
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
// that: a step 0.8% longer at 64^3, 1.3% at 256^3, a snapshot at 128^3 2.7%.
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

// (270 t1 - 27 t2 + 2 t3) / 64, |t| < 2^60, without overflow; where that is no
// whole number, the odd one next to it (odd in t, and the rounding to 53 bits that
// follows is that of the fraction)
__device__ __forceinline__ int64_t weigh_lap(int64_t t1, int64_t t2, int64_t t3) {
    const int64_t lo = (int64_t)((uint64_t)(uint32_t)t1 * 270u + (uint64_t)(uint32_t)t3 * 2u) -
                       (int64_t)((uint64_t)(uint32_t)t2 * 27u);
    const int64_t hi = (int64_t)(int32_t)(t1 >> 32) * 270 + (int64_t)(int32_t)(t3 >> 32) * 2 -
                       (int64_t)(int32_t)(t2 >> 32) * 27 + (lo >> 32);
    return (hi << 26) | (int64_t)((uint32_t)lo >> 6) | (int64_t)(((uint32_t)lo & 63u) != 0u);
}

// gradient and Laplacian, all values aligned to one exponent
template <bool NEAREST>
__device__ __forceinline__ void grad_lap(double f0, const double (&f)[3][6], uint32_t e, double* r) {
    const int64_t i0 = align<NEAREST>(f0, e);
    int64_t T[3] = {-6 * i0, -6 * i0, -6 * i0};
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        int64_t D[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int64_t u = align<NEAREST>(f[ax][d], e), w = align<NEAREST>(f[ax][d + 3], e);
            D[d] = u - w;
            T[d] += u + w;
        }
        r[ax] = to_double(weigh_grad(D[0], D[1], D[2]), e, 0);
    }
    r[3] = to_double(weigh_lap(T[0], T[1], T[2]), e, 6);
}

// the neighbours [+1, +2, +3, -1, -2, -3] of *p, index q of n
__device__ __forceinline__ void line(const double* p, int q, int n, int stride, double* f) {
#pragma unroll
    for (int d = 1; d <= 3; ++d) {
        f[d - 1] = __ldg(p + (q + d < n ? d : d - n) * stride);
        f[d + 2] = __ldg(p + (q >= d ? -d : n - d) * stride);
    }
}

// Where the stencil holds a zero, at (i, j, k) of nx, ny, nz: out of line, so that
// its instructions do not lie between those of the other sites (in line: 3%
// more per step at 256^3).
static __device__ __noinline__ void grad_lap_zero(const double* p, int i, int j, int k, int nx, int ny, int nz,
                                                  uint32_t e, double* r) {
    double f[3][6];
    line(p, i, nx, 1, f[0]);
    line(p, j, ny, nx, f[1]);
    line(p, k, nz, nx * ny, f[2]);
    grad_lap<true>(__ldg(p), f, e, r);
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
    // index and side along z; in a slab none that wrap (ghost planes)
    __device__ __forceinline__ int kz() const { return g.zg ? 1 << 29 : k; }
    __device__ __forceinline__ int nz() const { return g.zg ? 1 << 30 : g.nz; }
    // the neighbours of *p along an axis
    __device__ __forceinline__ void along(const double* p, int ax, double* f) const {
        int q = ax == 0 ? i : (ax == 1 ? j : kz());
        asm volatile("" : "+r"(q));  // keeps the offsets from being hoisted out of the caller's loop
        fix::line(p, q, ax == 0 ? g.nx : (ax == 1 ? g.ny : nz()), ax == 0 ? 1 : (ax == 1 ? g.nx : g.nx * g.ny), f);
    }
    __device__ __forceinline__ void grad_lap(int a, double& gx, double& gy, double& gz, double& lap) const {
        const double* p = at(a);
        double f[3][6];
        const double f0 = __ldg(p);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(p, ax, f[ax]);
        uint32_t e = fix::exp20(f0), lo = e;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) e = max(e, fix::largest(f[ax], lo));
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
        double r[4];
        if (lo != 0u)
            fix::grad_lap<false>(f0, f, e, r);
        else
            fix::grad_lap_zero(p, i, j, kz(), g.nx, g.ny, nz(), e, r);
        gx = r[0];
        gy = r[1];
        gz = r[2];
        lap = r[3];
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
