// stage_dd.cu -- DF64 form: the FP64 form's stage kernels (stage.cu) with
// every stencil, flux and RK4 combination evaluated in double-float
// arithmetic (dd.cuh) on the FP32 pipes.
//
// The state, the RK4 accumulator and the stage inputs keep the FP64 form's
// buffers and scheme (y, yn, xa, xb, [36][S] of 8 bytes, the reference's
// yn accumulation order, main_rk4.jl:6146-6437), each value stored as the
// float pair (hi, lo).  State I/O converts from / to FP64 exactly
// representable splits (hi = fl(v), lo = fl(v - hi)).
#include <algorithm>

#include "accessors.cuh"
#include "convert.cuh"
#include "dd.cuh"
#include "dd2.cuh"

namespace {

template <int REG>
struct DdBudget;
template <>
struct DdBudget<0> { static constexpr int kThreads = 128, kMinBlocks = 1; };
template <>
struct DdBudget<1> { static constexpr int kThreads = 128, kMinBlocks = 4; };
template <>
struct DdBudget<2> { static constexpr int kThreads = 128, kMinBlocks = 3; };

// Stencil sums in double-float with lazy normalisation: each partial sum is
// an unnormalised pair (h, l), h + l the value, |l| a few ulp of h at most.
// An addition is Knuth's TwoSum on the high parts plus the low parts (8
// FP32 operations); a product by a coefficient is the FMA product error
// plus the cross terms (4).  Only a finished derivative is renormalised
// (FastTwoSum, 3), where dd's operators renormalise after every operation
// (11 and 7).  The error per operation stays ~2^-47 of the operands.
struct Lz {
    float h, l;
};
__device__ __forceinline__ Lz lz_add(const Lz& a, const Lz& b) {
    const float s = a.h + b.h;
    const float v = s - a.h;
    const float e = (a.h - (s - v)) + (b.h - v);
    return Lz{s, e + (a.l + b.l)};
}
__device__ __forceinline__ Lz lz_sub(const Lz& a, const Lz& b) { return lz_add(a, Lz{-b.h, -b.l}); }
__device__ __forceinline__ Lz lz_mul(const dd& c, const Lz& x) {
    const float p = c.hi * x.h;
    float e = fmaf(c.hi, x.h, -p);
    e = fmaf(c.hi, x.l, e);
    e = fmaf(c.lo, x.h, e);
    return Lz{p, e};
}
__device__ __forceinline__ dd lz_done(const Lz& x) { return dd_fast_two_sum(x.h, x.l); }

// The stencil evaluations are out-of-line calls: the double-float stage is
// instruction-fetch bound (~20 k straight-line instructions per site), and
// one copy of each stencil routine replaces 16 + 4 + 4 inlined copies.
struct DdAcc : SiteAcc<float2, dd, SrcPtr36<float2>> {
    using Base = SiteAcc<float2, dd, SrcPtr36<float2>>;
    __device__ __forceinline__ Lz lz(int a, int off) const {
        const float2 v = __ldg(src.arr(a) + (c + off));
        return Lz{v.x, v.y};
    }
    // derivative along one axis (offsets o) in unnormalised form
    __device__ __forceinline__ Lz d1_lz(int a, const int* o) const {
        Lz g = lz_mul(s.a1, lz_sub(lz(a, o[0]), lz(a, o[3])));
        g = lz_add(g, lz_mul(s.a2, lz_sub(lz(a, o[1]), lz(a, o[4]))));
        return lz_add(g, lz_mul(s.a3, lz_sub(lz(a, o[2]), lz(a, o[5]))));
    }
    __device__ __noinline__ void grad_lap(int a, dd& gx, dd& gy, dd& gz, dd& lap) const {
        Lz S[3];  // sum over the axes of f(+k) + f(-k), k = 1, 2, 3
        const int* os[3] = {ox, oy, oz};
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const int* o = os[ax];
            Lz g;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const Lz p = lz(a, o[k]), m = lz(a, o[k + 3]);
                const dd& ck = k == 0 ? s.a1 : (k == 1 ? s.a2 : s.a3);
                const Lz t = lz_mul(ck, lz_sub(p, m));
                g = k == 0 ? t : lz_add(g, t);
                const Lz q = lz_add(p, m);
                S[k] = ax == 0 ? q : lz_add(S[k], q);
            }
            (ax == 0 ? gx : (ax == 1 ? gy : gz)) = lz_done(g);
        }
        Lz L = lz_mul(s.l0, lz(a, 0));
        L = lz_add(L, lz_mul(s.l1, S[0]));
        L = lz_add(L, lz_mul(s.l2, S[1]));
        lap = lz_done(lz_add(L, lz_mul(s.l3, S[2])));
    }
    __device__ __noinline__ void grad(int a, dd& gx, dd& gy, dd& gz) const {
        gx = lz_done(d1_lz(a, ox));
        gy = lz_done(d1_lz(a, oy));
        gz = lz_done(d1_lz(a, oz));
    }
    __device__ __noinline__ dd div3(int a) const {
        return lz_done(lz_add(lz_add(d1_lz(a, ox), d1_lz(a + 1, oy)), d1_lz(a + 2, oz)));
    }
};

template <int STAGE>
struct DdSink {
    const DdAcc& A;
    const float2* __restrict__ y;
    float2* yn;
    float2* __restrict__ xn;
    float2* acc_out;
    int64_t S;
    dd w, h;
    float2* cur;  // [12][S] Higgs currents of kt W and kt Y, from the first launch of a split stage to the others
    __device__ __forceinline__ void keep_current(int q, dd v) const { cur[q * S + A.c] = v.f2(); }
    __device__ __forceinline__ dd load_current(int q) const { return dd(__ldg(cur + q * S + A.c)); }
    __device__ __forceinline__ void operator()(int a, dd r) const {
        const int64_t q = a * S + A.c;
        if (STAGE == 1) {
            const dd ya = A.v(a);  // X1 == y
            yn[q] = (ya + w * r).f2();
            xn[q] = (ya + h * r).f2();
        } else if (STAGE < 4) {
            // read then written by this thread only: read-only path is safe
            yn[q] = (dd(__ldg(yn + q)) + w * r).f2();
            xn[q] = (dd(__ldg(y + q)) + h * r).f2();
        } else {
            acc_out[q] = (dd(__ldg(yn + q)) + w * r).f2();
        }
    }
};

Ptr36 pack8(const void* base, int64_t S) {
    Ptr36 P;
    for (int a = 0; a < 36; ++a) P.p[a] = static_cast<const char*>(base) + (size_t)a * S * 8;
    return P;
}

// PART (site_rates): 0 the whole stage; 1-3 its three parts (Higgs; SU(2);
// fields, auxiliaries and U(1)), launched one after the other when there
// are no beta terms.  The double-float stage is instruction-fetch bound
// (~20 k straight-line instructions per site): each part is a third of the
// code, and the stencil routines are shared out-of-line calls.
template <int STAGE, bool BETA, int REG, int PART>
__global__ void __launch_bounds__(DdBudget<REG>::kThreads, DdBudget<REG>::kMinBlocks)
    k_stage_dd(Grid g, const __grid_constant__ Ptr36 X, const float2* __restrict__ y, float2* yn,
               float2* __restrict__ xn, float2* acc_out, PhysCoef<dd> pc, StencilCoef<dd> sc, dd w, dd h,
               float2* cur) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= g.nx || j >= g.ny) return;
    DdAcc A{{{X}}};
    A.place(i, j, k, g.nx, g.ny, g.nz);
    A.s = sc;
    DdSink<STAGE> out{A, y, yn, xn, acc_out, g.S, w, h, cur};
    site_rates<dd, BETA, DdAcc, DdSink<STAGE>, PART>(A, pc, out);
}

// ------------------------------------------------- two sites per thread
// Even rows without beta terms, lattices whose pairs fill the SMs (384 threads
// each; 24^3 0.19 ms per step with one site per thread, 0.24 with two): thread = the x-adjacent sites (i0, i0 + 1), i0
// even, on packed double-float pairs (dd2.cuh), three launches per stage as
// above.  The arrays then hold a site pair as (hi0, hi1, lo0, lo1), one
// 16-byte load; the conversions read and write that order.
struct Dd2Acc {
    const float4* x;  // [36][S / 2]
    int64_t Sp;       // S / 2
    int c;            // pair index
    int ox[4];        // pairs at i0 - 4, i0 - 2, i0 + 2, i0 + 4
    int oy[6], oz[6];
    StencilCoef<dd2> s;

    __device__ __forceinline__ dd2 at(const float4* p, int off) const { return dd2(__ldg(p + off)); }
    __device__ __forceinline__ dd2 v(int a) const { return at(x + a * Sp + c, 0); }
    __device__ __forceinline__ static dd2 odd(const dd2& l, const dd2& r) {
        return dd2(make_float2(l.hi.y, r.hi.x), make_float2(l.lo.y, r.lo.x));
    }
    // neighbours +1, +2, +3, -1, -2, -3 along an axis
    __device__ __forceinline__ void along(const float4* p, int ax, dd2* f) const {
        if (ax == 0) {
            const dd2 qm2 = at(p, ox[0]), qm1 = at(p, ox[1]), q0 = at(p, 0), qp1 = at(p, ox[2]), qp2 = at(p, ox[3]);
            f[0] = odd(q0, qp1);
            f[1] = qp1;
            f[2] = odd(qp1, qp2);
            f[3] = odd(qm1, q0);
            f[4] = qm1;
            f[5] = odd(qm2, qm1);
        } else {
            const int* o = ax == 1 ? oy : oz;
#pragma unroll
            for (int k = 0; k < 6; ++k) f[k] = at(p, o[k]);
        }
    }
    __device__ __forceinline__ dd2 weigh(const dd2* f) const {
        return mul2(s.a1, f[0] - f[3]) + mul2(s.a2, f[1] - f[4]) + mul2(s.a3, f[2] - f[5]);
    }
    __device__ __forceinline__ dd2 weigh_lap(const dd2& f0, const dd2* S) const {
        return mul2(s.l0, f0) + mul2(s.l1, S[0]) + mul2(s.l2, S[1]) + mul2(s.l3, S[2]);
    }
    __device__ __noinline__ void grad_lap(int a, dd2& gx, dd2& gy, dd2& gz, dd2& lap) const {
        const float4* p = x + a * Sp + c;
        dd2 S[3], f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(p, ax, f[ax]);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            (ax == 0 ? gx : (ax == 1 ? gy : gz)) = done2(weigh(f[ax]));
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const dd2 q = f[ax][k] + f[ax][k + 3];
                S[k] = ax == 0 ? q : S[k] + q;
            }
        }
        lap = done2(weigh_lap(at(p, 0), S));
    }
    __device__ __noinline__ dd2 lap(int a) const {
        const float4* p = x + a * Sp + c;
        dd2 S[3], f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(p, ax, f[ax]);
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const dd2 q = f[ax][k] + f[ax][k + 3];
                S[k] = ax == 0 ? q : S[k] + q;
            }
        }
        return done2(weigh_lap(at(p, 0), S));
    }
    __device__ __noinline__ dd2 d1(int a, int ax) const {
        dd2 f[6];
        along(x + a * Sp + c, ax, f);
        return done2(weigh(f));
    }
    __device__ __noinline__ void grad(int a, dd2& gx, dd2& gy, dd2& gz) const {
        dd2 f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(x + a * Sp + c, ax, f[ax]);
        gx = done2(weigh(f[0]));
        gy = done2(weigh(f[1]));
        gz = done2(weigh(f[2]));
    }
    __device__ __noinline__ dd2 div3(int a) const {
        dd2 f[3][6];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) along(x + (a + ax) * Sp + c, ax, f[ax]);
        return done2(weigh(f[0]) + weigh(f[1]) + weigh(f[2]));
    }

    __device__ __forceinline__ void place(int ip, int j, int k, int npx, int ny, int nz) {
        c = ip + npx * (j + ny * k);
        ox[0] = ip >= 2 ? -2 : npx - 2;
        ox[1] = ip >= 1 ? -1 : npx - 1;
        ox[2] = ip + 1 < npx ? 1 : 1 - npx;
        ox[3] = ip + 2 < npx ? 2 : 2 - npx;
        axis_offsets(j, ny, npx, oy);
        axis_offsets(k, nz, npx * ny, oz);
    }
};

template <int STAGE>
struct Dd2Sink {
    const Dd2Acc& A;
    const float4* __restrict__ y;
    float4* yn;
    float4* xn;
    dd2 w, h;
    float4* cur;  // [12][S / 2] Higgs currents, as DdSink::cur
    __device__ __forceinline__ void keep_current(int q, const dd2& v) const { cur[q * A.Sp + A.c] = done2(v).f4(); }
    __device__ __forceinline__ dd2 load_current(int q) const { return dd2(__ldg(cur + q * A.Sp + A.c)); }
    __device__ __forceinline__ void operator()(int a, const dd2& rate) const {
        const int64_t q = a * A.Sp + A.c;
        const dd2 r = done2(rate);
        if (STAGE < 4) {
            // read then written by this thread only: read-only path is safe
            const dd2 ya = STAGE == 1 ? A.v(a) : dd2(__ldg(y + q));  // X1 == y
            yn[q] = done2((STAGE == 1 ? ya : dd2(__ldg(yn + q))) + w * r).f4();
            xn[q] = done2(ya + h * r).f4();
        } else {
            xn[q] = done2(dd2(__ldg(yn + q)) + w * r).f4();  // the new y
        }
    }
};

template <int STAGE, int REG, int PART>
__global__ void __launch_bounds__(DdBudget<REG>::kThreads, DdBudget<REG>::kMinBlocks)
    k_stage_dd2(Grid g, const float4* __restrict__ X, const float4* __restrict__ y, float4* yn, float4* xn,
                const __grid_constant__ PhysCoef<dd2> pc, const __grid_constant__ StencilCoef<dd2> sc, dd2 w, dd2 h,
                float4* cur, Walk walk) {
    int ip, j, k;
    const int npx = g.nx >> 1;
    if (!walk.site(npx, g.ny, g.nz, ip, j, k)) return;
    Dd2Acc A;
    A.x = X;
    A.Sp = g.S >> 1;
    A.place(ip, j, k, npx, g.ny, g.nz);
    A.s = sc;
    Dd2Sink<STAGE> out{A, y, yn, xn, w, h, cur};
    if constexpr (PART == 1)
        higgs_rates_by_axis<dd2>(A, pc, out);
    else
        site_rates<dd2, false, Dd2Acc, Dd2Sink<STAGE>, PART>(A, pc, out);
}

template <int STAGE, int REG>
void stage_dd2(const Grid& g, const Tiling& t, cudaStream_t st, const double* X, double* y, double* yn, double* xn,
               const PhysCoef<dd2>& pc, const StencilCoef<dd2>& sc, dd2 w, dd2 h, double* cur) {
    dim3 gr, bl;
    const Walk walk = fp32_walk(g.nx / 2, g.ny, g.nz, t, true, gr, bl);
    auto f = [](const double* v) { return reinterpret_cast<float4*>(const_cast<double*>(v)); };
    k_stage_dd2<STAGE, REG, 1><<<gr, bl, 0, st>>>(g, f(X), f(y), f(yn), f(xn), pc, sc, w, h, f(cur), walk);
    k_stage_dd2<STAGE, REG, 2><<<gr, bl, 0, st>>>(g, f(X), f(y), f(yn), f(xn), pc, sc, w, h, f(cur), walk);
    k_stage_dd2<STAGE, REG, 3><<<gr, bl, 0, st>>>(g, f(X), f(y), f(yn), f(xn), pc, sc, w, h, f(cur), walk);
}

template <int REG>
void step_dd2(const Grid& g, const Tiling& t, double* y, double* yn, double* xa, double* xb, double* cur,
              const ewpt_params& p, double Jex, double gam, cudaStream_t st) {
    const PhysCoef<dd2> pc = make_phys<dd2>(p, Jex, gam);
    const StencilCoef<dd2> sc = make_stencil<dd2>(p.dx);
    const dd2 w6(p.dt / 6.), w3(p.dt / 3.), h2(p.dt / 2.), h1(p.dt), z(0.0);
    stage_dd2<1, REG>(g, t, st, y, y, yn, xa, pc, sc, w6, h2, cur);
    stage_dd2<2, REG>(g, t, st, xa, y, yn, xb, pc, sc, w3, h2, cur);
    stage_dd2<3, REG>(g, t, st, xb, y, yn, xa, pc, sc, w3, h1, cur);
    stage_dd2<4, REG>(g, t, st, xa, y, yn, y, pc, sc, w6, z, cur);
}

// The same conversions for arrays in site pairs: S even, a thread per pair.
__global__ void __launch_bounds__(256) k_to_dd2(int64_t Sp, const __grid_constant__ Ptr36 src, float4* pairs) {
    const double* v = reinterpret_cast<const double*>(src.p[blockIdx.y]);
    float4* out = pairs + blockIdx.y * Sp;
#pragma unroll 2
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < Sp; q += (int64_t)gridDim.x * blockDim.x) {
        const double a = v[2 * q], b = v[2 * q + 1];
        float4 f;
        split_f64(a, f.x, f.z);
        split_f64(b, f.y, f.w);
        out[q] = f;
    }
}

__global__ void __launch_bounds__(256) k_from_dd2(int64_t Sp, const float4* __restrict__ pairs,
                                                  const __grid_constant__ MPtr36 dst) {
    const float4* in = pairs + blockIdx.y * Sp;
    double* out = reinterpret_cast<double*>(dst.p[blockIdx.y]);
#pragma unroll 2
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < Sp; q += (int64_t)gridDim.x * blockDim.x) {
        const float4 f = __ldg(in + q);
        out[2 * q] = join_f64(f.x, f.z);
        out[2 * q + 1] = join_f64(f.y, f.w);
    }
}

// FP64 arrays <-> float pairs (convert.cuh), array blockIdx.y; in place when
// the pairs lie over the array itself, each element by one thread.  Bound by
// memory: 1.2 GB at 128^3; with C casts k_to_dd / k_from_dd took 557 / 411 us
// there, the time of their FP64-pipe instructions.
__global__ void __launch_bounds__(256) k_to_dd(int64_t S, const __grid_constant__ Ptr36 src, float2* pairs) {
    const double* v = reinterpret_cast<const double*>(src.p[blockIdx.y]);
    float2* out = pairs + blockIdx.y * S;
#pragma unroll 4
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < S; q += (int64_t)gridDim.x * blockDim.x) {
        float2 f;
        split_f64(v[q], f.x, f.y);
        out[q] = f;
    }
}

__global__ void __launch_bounds__(256) k_from_dd(int64_t S, const float2* __restrict__ pairs,
                                                 const __grid_constant__ MPtr36 dst) {
    const float2* in = pairs + blockIdx.y * S;
    double* out = reinterpret_cast<double*>(dst.p[blockIdx.y]);
#pragma unroll 4
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < S; q += (int64_t)gridDim.x * blockDim.x) {
        const float2 v = __ldg(in + q);
        out[q] = join_f64(v.x, v.y);
    }
}

dim3 pair_grid(int64_t S, int arrays) { return dim3((unsigned)std::min<int64_t>((S + 1023) / 1024, 4096), arrays); }

// One stage: the whole stage with beta terms, else its three parts.
template <int STAGE, bool BETA, int REG>
void stage_dd(const dim3& gr, const dim3& bl, cudaStream_t st, const Grid& g, const float2* X, const float2* y,
              float2* yn, float2* xn, float2* acc_out, const PhysCoef<dd>& pc, const StencilCoef<dd>& sc, dd w,
              dd h, float2* cur) {
    const Ptr36 P = pack8(X, g.S);
    if constexpr (BETA) {
        k_stage_dd<STAGE, true, REG, 0><<<gr, bl, 0, st>>>(g, P, y, yn, xn, acc_out, pc, sc, w, h, cur);
    } else {
        k_stage_dd<STAGE, false, REG, 1><<<gr, bl, 0, st>>>(g, P, y, yn, xn, acc_out, pc, sc, w, h, cur);
        k_stage_dd<STAGE, false, REG, 2><<<gr, bl, 0, st>>>(g, P, y, yn, xn, acc_out, pc, sc, w, h, cur);
        k_stage_dd<STAGE, false, REG, 3><<<gr, bl, 0, st>>>(g, P, y, yn, xn, acc_out, pc, sc, w, h, cur);
    }
}

template <bool BETA, int REG>
void step_dd(const Grid& g, const Tiling& t, float2* y, float2* yn, float2* xa, float2* xb, const PhysCoef<dd>& pc,
             const StencilCoef<dd>& sc, double dt, float2* cur, cudaStream_t st) {
    const dim3 gr((g.nx + t.bx - 1) / t.bx, (g.ny + t.by - 1) / t.by, g.nz), bl(t.bx, t.by);
    const dd w6(dt / 6.), w3(dt / 3.), h2(dt / 2.), h1(dt), z(0.0);
    stage_dd<1, BETA, REG>(gr, bl, st, g, y, y, yn, xa, nullptr, pc, sc, w6, h2, cur);
    stage_dd<2, BETA, REG>(gr, bl, st, g, xa, y, yn, xb, nullptr, pc, sc, w3, h2, cur);
    stage_dd<3, BETA, REG>(gr, bl, st, g, xb, y, yn, xa, nullptr, pc, sc, w3, h1, cur);
    stage_dd<4, BETA, REG>(gr, bl, st, g, xa, y, yn, nullptr, y, pc, sc, w6, z, cur);
}

template <bool BETA>
void step_dd_r(const Grid& g, const Tiling& t, float2* y, float2* yn, float2* xa, float2* xb, const PhysCoef<dd>& pc,
               const StencilCoef<dd>& sc, double dt, float2* cur, cudaStream_t st) {
    // the 128-register variant spills heavily in this form and runs as variant 0
    if (t.reg == 2)
        step_dd<BETA, 2>(g, t, y, yn, xa, xb, pc, sc, dt, cur, st);
    else
        step_dd<BETA, 0>(g, t, y, yn, xa, xb, pc, sc, dt, cur, st);
}

}  // namespace

cudaError_t launch_step_dd(const Grid& g, const Tiling& t, double* y, double* yn, double* xa, double* xb,
                           double* cur, const ewpt_params& p, double Jex, double gam, cudaStream_t st) {
    if (dd_in_pairs(g, p)) {
        // 128 registers run fastest (256^3: 45.8 ms per step against 48.2 with
        // 168 and 55.9 with 255)
        if (t.reg == 0 && !t.pick)
            step_dd2<0>(g, t, y, yn, xa, xb, cur, p, Jex, gam, st);
        else if (t.reg == 2)
            step_dd2<2>(g, t, y, yn, xa, xb, cur, p, Jex, gam, st);
        else
            step_dd2<1>(g, t, y, yn, xa, xb, cur, p, Jex, gam, st);
        return cudaGetLastError();
    }
    const PhysCoef<dd> pc = make_phys<dd>(p, Jex, gam);
    const StencilCoef<dd> sc = make_stencil<dd>(p.dx);
    auto f2p = [](double* v) { return reinterpret_cast<float2*>(v); };
    if (p.beta_w != 0.0 || p.beta_y != 0.0)
        step_dd_r<true>(g, t, f2p(y), f2p(yn), f2p(xa), f2p(xb), pc, sc, p.dt, f2p(cur), st);
    else
        step_dd_r<false>(g, t, f2p(y), f2p(yn), f2p(xa), f2p(xb), pc, sc, p.dt, f2p(cur), st);
    return cudaGetLastError();
}

bool dd_in_pairs(const Grid& g, const ewpt_params& p) {
    return g.nx % 2 == 0 && p.beta_w == 0.0 && p.beta_y == 0.0 && g.S > 152 * 768;
}

cudaError_t launch_to_dd(int64_t S, bool in_pairs, const Ptr36& src, double* pairs, cudaStream_t st) {
    if (in_pairs)
        k_to_dd2<<<pair_grid(S / 2, 36), 256, 0, st>>>(S / 2, src, reinterpret_cast<float4*>(pairs));
    else
        k_to_dd<<<pair_grid(S, 36), 256, 0, st>>>(S, src, reinterpret_cast<float2*>(pairs));
    return cudaGetLastError();
}

cudaError_t launch_from_dd(int64_t S, bool in_pairs, const double* pairs, const MPtr36& dst, cudaStream_t st, int arrays) {
    if (in_pairs)
        k_from_dd2<<<pair_grid(S / 2, arrays), 256, 0, st>>>(S / 2, reinterpret_cast<const float4*>(pairs), dst);
    else
        k_from_dd<<<pair_grid(S, arrays), 256, 0, st>>>(S, reinterpret_cast<const float2*>(pairs), dst);
    return cudaGetLastError();
}
