// stage_fp64.cuh -- one site of the FP64 form's 6th-order stages: the stencils and
// the roles of the four warps that share it (stage_fp64.cu).  A host compiler
// takes this file too, with the warps as threads (oracle/devstage.cc).
#pragma once
#include <type_traits>

#include "accessors.cuh"
#include "fixstencil.cuh"

namespace {

// Couplings for derivatives in units of t = 1/(60 dx) and Laplacians of
// 1/(180 dx^2): a sum that holds a derivative is in units of t, and the last
// factor of its rate restores it.
struct Coef {
    double it, t;              // 1/t, t
    double ryw, igw;           // g'/g, 1/g
    double hgw, gw;            // g/2, g where a product meets a derivative: over t
    double omgp2, gg, ggy;     // (1 - gp2) t; gp2 g, gp2 g'
    double lam2h, vev2, hJexh, gamh;  // 2 lambda, Jex/2 and gamma over t g/2; vev^2
    double hgw_o, gw_o, gy_o;  // t g/2, t g, t g': end a rate
    double lap_h, lap_w, lap_y;
    double bW, bY, bW2, bY2;   // beta_W, beta_Y and their doubles, times t
};

Coef make_coef(const ewpt_params& p, double Jex, double gam) {
    const PhysCoef<double> f = make_phys<double>(p, Jex, gam);
    const double T = 60.0 * p.dx, iU = 1.0 / (180.0 * p.dx * p.dx);
    Coef c;
    c.it = T;
    c.t = 1.0 / T;
    c.ryw = f.ryw;
    c.igw = f.igw;
    c.hgw = T * f.hgw;
    c.gw = T * f.gw;
    c.omgp2 = f.omgp2 / T;
    c.gg = f.gg;
    c.ggy = f.ggy;
    c.lam2h = f.lam2h * T;
    c.vev2 = f.vev2;
    c.hJexh = f.hJexh * T;
    c.gamh = f.gamh * T;
    c.hgw_o = f.hgw / T;
    c.gw_o = f.gw / T;
    c.gy_o = f.gy / T;
    c.lap_h = iU / c.hgw_o;
    c.lap_w = iU / c.gw_o;
    c.lap_y = iU;
    c.bW = f.bW / T;
    c.bY = f.bY / T;
    c.bW2 = f.bW2 / T;
    c.bY2 = f.bY2 / T;
    return c;
}

constexpr int kSites = 32, kWarps = 4;
constexpr int kSlots = 80;  // d_i of arrays 0-19 (3 a + i), Laplacians of 0-15 (60 + a), divergences (76 + c)

struct Shared {
    double s[kSlots][kSites];
    double j[12][kSites];  // currents J^a_i (3 a + i) and J^Y_i (9 + i), in units of g t, g' t
    // axis i's part of the rate of Higgs component b: in place of d_i phi_b
    __device__ __forceinline__ double& part(int b, int i, int lane) { return s[3 * b + i][lane]; }
};
struct SharedBeta : Shared {
    double f[9][kSites];   // F^a_xy, F^a_xz, F^a_yz (3 a + m)
    double h[12][kSites];  // the axes' parts: the colours still need d phi
    __device__ __forceinline__ double& part(int b, int i, int lane) { return h[3 * b + i][lane]; }
};
template <bool BETA>
using SharedOf = std::conditional_t<BETA, SharedBeta, Shared>;

struct StageSink {
    const double* y;
    double* yn;
    double* xn;  // next stage input, or the new y (stage 4)
    int64_t S;
    double w[3], h[3];  // by unit
};

// Units of the rates handed over: 1, Coef::hgw_o and Coef::gw_o.  The last two
// are in the sink's weights, one multiplication less for 13 arrays.
enum Unit { kOne, kHiggs, kGauge };

// the rate of array a at the site c; x: the stage input's value (stage 1)
template <int STAGE, Unit U = kOne>
__device__ __forceinline__ void put(const StageSink& o, int a, int c, bool live, double x, double r) {
    if (!live) return;
    const int64_t q = a * o.S + c;
    if (STAGE == 1) {  // X1 == y
        o.yn[q] = fma(r, o.w[U], x);
        o.xn[q] = fma(r, o.h[U], x);
    } else if (STAGE < 4) {
        // read then written by this thread only: the read-only path lets these
        // loads issue ahead of earlier stores
        o.yn[q] = fma(r, o.w[U], __ldg(o.yn + q));
        o.xn[q] = fma(r, o.h[U], __ldg(o.y + q));
    } else {
        o.xn[q] = fma(r, o.w[U], __ldg(o.yn + q));
    }
}
struct RatesOut {
    MPtr36 R;
    double unit[3];
};
template <int STAGE, Unit U = kOne>
__device__ __forceinline__ void put(const RatesOut& o, int a, int c, bool live, double, double r) {
    if (live) reinterpret_cast<double*>(o.R.p[a])[c] = U == kOne ? r : o.unit[U] * r;
}

// Named barriers.  1: the colour warps' parts of the Higgs rates are in shared
// memory; only the Higgs warp waits.  2: the currents and every colour's E_ij
// are; the three colour warps wait.
// (A host compiler's caller defines them.)
#ifdef __CUDACC__
__device__ __forceinline__ void parts_written() {
    asm volatile("bar.arrive 1, %0;" ::"n"(kSites * kWarps) : "memory");
}
__device__ __forceinline__ void parts_ready() { asm volatile("bar.sync 1, %0;" ::"n"(kSites * kWarps) : "memory"); }
__device__ __forceinline__ void colours_ready() {
    asm volatile("bar.sync 2, %0;" ::"n"(kSites * (kWarps - 1)) : "memory");
}
#else
void parts_written();
void parts_ready();
void colours_ready();
#endif

// The derivatives and the field strength of a colour act on the other two only
// as E_ij = F_ij - d_j W_i: replaces d_j W^a_i (i != j) by E_ij, u = W^{a+1}, v =
// W^{a+2}; F_xy, F_xz, F_yz to F.
__device__ __forceinline__ void strengths(Shared& sh, int lane, int a, const double* u, const double* v, double gw,
                                          double* F) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        const int i = m == 2 ? 1 : 0, j = m == 0 ? 1 : 2;
        double &dij = sh.s[3 * (4 + 3 * a + i) + j][lane], &dji = sh.s[3 * (4 + 3 * a + j) + i][lane];
        F[m] = dji - dij + gw * (u[i] * v[j] - u[j] * v[i]);  // d_i W_j - d_j W_i + g (...)
        const double e = -F[m] - dji;
        dij = F[m] - dij;
        dji = e;
    }
}

// Q_i += sum_j f_j E^b_ij (E_ii = -d_i W_i), or -= with NEG
template <bool NEG>
__device__ __forceinline__ void add_strengths(const Shared& sh, int lane, int b, const double* f, double* Q) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double e = sh.s[3 * (4 + 3 * b + i) + j][lane];
            Q[i] = (i == j) != NEG ? fma(-f[j], e, Q[i]) : fma(f[j], e, Q[i]);
        }
}

// Axis i's terms of the covariant Higgs equation: the currents along i and
// W_i (d_i phi + D_i phi) for each component.
template <bool BETA>
__device__ __forceinline__ void axis_part(const FixAcc& A, const Coef& c, SharedOf<BETA>& sh, int lane,
                                          int i) {
    const double p[4] = {A.v(0), A.v(1), A.v(2), A.v(3)};
    const double W1 = A.v(4 + i), W2 = A.v(7 + i), W3 = A.v(10 + i), Yr = c.ryw * A.v(13 + i);
    const double Zp = W3 + Yr, Zm = W3 - Yr;
    double d1 = sh.s[i][lane], d2 = sh.s[3 + i][lane], d3 = sh.s[6 + i][lane], d4 = sh.s[9 + i][lane];
    double D1, D2, D3, D4;
    cov_deriv_s(d1, d2, d3, d4, p[0], p[1], p[2], p[3], W1, W2, Zp, Zm, c.hgw, D1, D2, D3, D4);
    sh.j[i][lane] = p[0] * D4 - p[1] * D3 + p[2] * D2 - p[3] * D1;
    sh.j[3 + i][lane] = -p[0] * D3 - p[1] * D4 + p[2] * D1 + p[3] * D2;
    const double j12 = p[0] * D2 - p[1] * D1, j34 = p[2] * D4 - p[3] * D3;
    sh.j[6 + i][lane] = j12 - j34;
    sh.j[9 + i][lane] = j12 + j34;
    d1 += D1;
    d2 += D2;
    d3 += D3;
    d4 += D4;
    sh.part(0, i, lane) = W1 * d4 - W2 * d3 + Zp * d2;
    sh.part(1, i, lane) = -W1 * d3 - W2 * d4 - Zp * d1;
    sh.part(2, i, lane) = W1 * d2 + W2 * d1 - Zm * d4;
    sh.part(3, i, lane) = W2 * d2 - W1 * d1 + Zm * d3;
}

template <int STAGE, bool BETA, class Out>
__device__ __forceinline__ void higgs_warp(const FixAcc& A, const Coef& c, SharedOf<BETA>& sh, int lane,
                                           bool live, const Out& out) {
    // k_field = momentum
#pragma unroll 4
    for (int f = 0; f < 16; ++f) put<STAGE>(out, f, A.c, live, STAGE == 1 ? A.v(f) : 0.0, A.v(20 + f));
    const double p[4] = {A.v(0), A.v(1), A.v(2), A.v(3)};
    const double pt[4] = {A.v(20), A.v(21), A.v(22), A.v(23)};
    const double qY = p[0] * pt[1] - p[1] * pt[0] + p[2] * pt[3] - p[3] * pt[2];
    put<STAGE>(out, 19, A.c, live, STAGE == 1 ? A.v(19) : 0.0, c.omgp2 * sh.s[79][lane] + c.ggy * qY);
    double a[4];
    {
        const double mag = p[0] * p[0] + p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
        const double potg = c.lam2h * (mag - c.vev2) + c.hJexh;
        // gamma / |Phi|^2, its 0/0 at |Phi| = 0 kept; no division without damping
        double damp = fix::zero_bits(mag) ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
        if (!fix::zero_bits(c.gamh)) damp = c.gamh / mag;
        const double G1 = c.it * A.v(16), G2 = c.it * A.v(17), G3 = c.it * A.v(18), S = c.it * A.v(19);
        const double q12 = G3 + c.ryw * S, q34 = c.ryw * S - G3;
        a[0] = q12 * p[1] - G2 * p[2] + G1 * p[3] - p[0] * (potg + damp * (p[0] * pt[0]));
        a[1] = -q12 * p[0] - G1 * p[2] - G2 * p[3] - p[1] * (potg + damp * (p[1] * pt[1]));
        a[2] = q34 * p[3] + G2 * p[0] + G1 * p[1] - p[2] * (potg + damp * (p[2] * pt[2]));
        a[3] = -q34 * p[2] - G1 * p[0] + G2 * p[1] - p[3] * (potg + damp * (p[3] * pt[3]));
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) a[b] += sh.s[60 + b][lane] * c.lap_h;
    parts_ready();
    double bsum = 0.0;
    if (BETA) {
        const auto& f = static_cast<SharedBeta&>(sh).f;  // written before the colours' arrival at the barrier
        // the reference pairs the y and z components of every colour with the
        // first colour's momenta (main_rk4.jl:350-352)
        const double E1y = A.v(25), E1z = A.v(26);
        double bWt = 0.0;
#pragma unroll
        for (int b = 0; b < 3; ++b)
            bWt += A.v(24 + 3 * b) * f[3 * b + 2][lane] - E1y * f[3 * b + 1][lane] + E1z * f[3 * b][lane];
        const double Fxy = sh.s[3 * 14][lane] - sh.s[3 * 13 + 1][lane], Fxz = sh.s[3 * 15][lane] - sh.s[3 * 13 + 2][lane],
                     Fyz = sh.s[3 * 15 + 1][lane] - sh.s[3 * 14 + 2][lane];
        bsum = c.bW * bWt + c.bY * (A.v(33) * Fyz - A.v(34) * Fxz + A.v(35) * Fxy);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const double r = a[b] + (sh.part(b, 0, lane) + sh.part(b, 1, lane) + sh.part(b, 2, lane));
        if (BETA)
            put<STAGE>(out, 20 + b, A.c, live, pt[b], c.hgw_o * r + bsum * p[b]);
        else
            put<STAGE, kHiggs>(out, 20 + b, A.c, live, pt[b], r);
    }
}

// colour a = 0, 1, 2 (and axis a)
template <int STAGE, bool BETA, class Out>
__device__ __forceinline__ void colour_warp(const FixAcc& A, const Coef& c, SharedOf<BETA>& sh, int lane,
                                            bool live, int a, const Out& out) {
    const int b = a == 2 ? 0 : a + 1, cc = a == 0 ? 2 : a - 1;
    axis_part<BETA>(A, c, sh, lane, a);
    double Wb[3], Wc[3], Q[3], F[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        Wb[i] = A.v(4 + 3 * b + i);
        Wc[i] = A.v(4 + 3 * cc + i);
    }
    strengths(sh, lane, a, Wb, Wc, c.gw, F);
    if (BETA)
#pragma unroll
        for (int m = 0; m < 3; ++m) static_cast<SharedBeta&>(sh).f[3 * a + m][lane] = F[m];
    parts_written();
    {
        // k_Gamma^a: Higgs charge p M_a pt, then -(W^b . Wt^c - W^c . Wt^b)
        const int i0 = a == 1 ? 2 : 0, i1 = a == 0 ? 3 : a == 1 ? 0 : 1, i2 = a == 0 ? 2 : 3, i3 = a == 2 ? 2 : 1;
        double q = A.v(i0) * A.v(20 + i1) - A.v(i1) * A.v(20 + i0) + A.v(i2) * A.v(20 + i3) - A.v(i3) * A.v(20 + i2);
#pragma unroll
        for (int i = 0; i < 3; ++i) q += Wc[i] * A.v(24 + 3 * b + i) - Wb[i] * A.v(24 + 3 * cc + i);
        put<STAGE>(out, 16 + a, A.c, live, STAGE == 1 ? A.v(16 + a) : 0.0,
                   c.omgp2 * sh.s[76 + a][lane] + c.gg * q);
    }
    const double Gb = c.it * A.v(16 + b), Gc = c.it * A.v(16 + cc);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        Q[i] = Wc[i] * Gb - Wb[i] * Gc + sh.s[60 + 4 + 3 * a + i][lane] * c.lap_w - sh.s[3 * (16 + a) + i][lane] * c.igw;
    colours_ready();
    add_strengths<false>(sh, lane, b, Wc, Q);
    add_strengths<true>(sh, lane, cc, Wb, Q);
    double kY = c.lap_y * sh.s[60 + 13 + a][lane] - c.t * sh.s[3 * 19 + a][lane];
    double kb[3] = {};  // beta terms
    if (BETA) {
        const double p[4] = {A.v(0), A.v(1), A.v(2), A.v(3)};
        double cv[3];
        const double pdot = A.v(20) * p[0] + A.v(21) * p[1] + A.v(22) * p[2] + A.v(23) * p[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            cv[i] = sh.s[i][lane] * p[0] + sh.s[3 + i][lane] * p[1] + sh.s[6 + i][lane] * p[2] + sh.s[9 + i][lane] * p[3];
        const double B[3] = {F[2], -F[1], F[0]};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int j = (i + 1) % 3, k = (i + 2) % 3;
            kb[i] = c.bW2 * (cv[j] * A.v(24 + 3 * a + k) - cv[k] * A.v(24 + 3 * a + j) - pdot * B[i]);
        }
        // component i = a of Y: dual field strength d_j Y_k - d_k Y_j
        const int j = b, k = cc;
        const double BY = sh.s[3 * (13 + k) + j][lane] - sh.s[3 * (13 + j) + k][lane];
        const double cj = a == 0 ? cv[1] : a == 1 ? cv[2] : cv[0], ck = a == 0 ? cv[2] : a == 1 ? cv[0] : cv[1];
        kY += c.bY2 * (cj * A.v(33 + k) - ck * A.v(33 + j) - pdot * BY);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int arr = 24 + 3 * a + i;
        const double r = Q[i] + sh.j[3 * a + i][lane];
        if (BETA)
            put<STAGE>(out, arr, A.c, live, STAGE == 1 ? A.v(arr) : 0.0, c.gw_o * r + kb[i]);
        else
            put<STAGE, kGauge>(out, arr, A.c, live, STAGE == 1 ? A.v(arr) : 0.0, r);
    }
    put<STAGE>(out, 33 + a, A.c, live, STAGE == 1 ? A.v(33 + a) : 0.0, kY + c.gy_o * sh.j[9 + a][lane]);
}

// warp's quarter of the stencils
__device__ __forceinline__ void stencils(const FixAcc& A, Shared& sh, int lane, int warp) {
#pragma unroll 1
    for (int n = 0; n < 4; ++n) {
        const int a = 4 * warp + n;
        double gx, gy, gz, l;
        A.grad_lap(a, gx, gy, gz, l);
        sh.s[3 * a][lane] = gx;
        sh.s[3 * a + 1][lane] = gy;
        sh.s[3 * a + 2][lane] = gz;
        sh.s[60 + a][lane] = l;
    }
    {
        const int a = 16 + warp;
        double gx, gy, gz;
        A.grad(a, gx, gy, gz);
        sh.s[3 * a][lane] = gx;
        sh.s[3 * a + 1][lane] = gy;
        sh.s[3 * a + 2][lane] = gz;
        sh.s[76 + warp][lane] = A.div3(24 + 3 * warp);
    }
}

}  // namespace
