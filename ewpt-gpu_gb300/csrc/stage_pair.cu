// stage_pair.cu -- FP32-form RK4 stage kernels with two sites per thread.
//
// Same stage structure and arithmetic as k_stage_fp32 (stage.cu; with s2 its
// roundings too), but each thread owns the x-adjacent sites (i0, i0+1), i0 even, and runs the physics
// on packed float pairs (f32x2.cuh): every flux operation is one FFMA2 /
// FADD2 / FMUL2 for both sites, and every neighbour access is a float2 load.
// For the x stencil the pairs at i0-4, i0-2, i0, i0+2, i0+4 (five aligned
// float2 loads) are re-paired into the +-1, +-2, +-3 neighbour pairs; y and z
// neighbours are aligned float2 loads of the same x pair.  The buffers use
// the ghosted layout (ewpt_internal.cuh), so neighbours past a face are read
// from the ghost cells along y and z (refreshed by k_ghost_fill_yz after each
// stage) and wrapped in the offsets along x.  Needs nx even.
#include <algorithm>

#include "accessors.cuh"
#include "physics_fp32.cuh"

namespace {

template <int REG>
struct PairBudget;
template <>
struct PairBudget<0> { static constexpr int kThreads = 128, kMinBlocks = 1; };
template <>
struct PairBudget<1> { static constexpr int kThreads = 128, kMinBlocks = 4; };
template <>
struct PairBudget<2> { static constexpr int kThreads = 128, kMinBlocks = 3; };

struct PairBufs {
    float* yhi;
    float* ylo;
    float* kacc;
};

// The scheme of Fp32Sink (stage.cu): no stored rate sum for the fields.
template <int STAGE, class Acc>
struct PairSink {
    using V = typename Acc::Value;
    const Acc& A;
    const Layout& L;
    PairBufs b;
    float* xn;
    V h, w6;
    const float *x2, *x3;  // stage 4: the inputs of stages 2 and 3
    __device__ __forceinline__ static float2* at(float* base, int64_t q) { return reinterpret_cast<float2*>(base + q); }
    __device__ __forceinline__ static float2 rd(const float* base, int64_t q) {
        return __ldg(reinterpret_cast<const float2*>(base + q));
    }
    __device__ __forceinline__ void operator()(int a, V r) const {
        const int64_t q = a * L.P + A.c;
        if (STAGE < 4) {
            // read then written by this thread only: read-only path is safe
            if (a >= 16) *at(b.kacc, q) = STAGE == 1 ? r.v : (V(rd(b.kacc, q)) + V(2.f) * r).v;
            float* x = STAGE == 3 && a >= 20 ? b.kacc - 20 * L.P : xn;  // X4's momenta
            *at(x, q) = ((STAGE == 1 ? A.v(a) : V(rd(b.yhi, q))) + h * r).v;
        } else {
            V k;
            if (a < 16) {
                const int64_t m = q + 20 * L.P;
                k = V(rd(b.yhi, m)) + V(2.f) * V(rd(x2, m));
                k = k + V(2.f) * V(rd(x3, m));
            } else {
                k = V(rd(b.kacc, q));
            }
            const V s = k + r;
            V hi(rd(b.yhi, q)), lo(rd(b.ylo, q));
            if constexpr (V::kFirst)
                acc_hilo(hi, lo, w6 * s);
            else
                acc_hilo(hi, lo, V(w6 * s));
            *at(b.yhi, q) = hi.v;
            *at(b.ylo, q) = lo.v;
        }
    }
};

__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// COMP: the compensated mode (gauge Laplacians and auxiliary gradients as
// compensated pairs, accessors.cuh PairAcc); scl = the coefficients' low parts.
// V = s2: the bits of k_stage_fp32.
template <int STAGE, bool BETA, int REG, bool COMP, class V>
__global__ void __launch_bounds__(PairBudget<REG>::kThreads, PairBudget<REG>::kMinBlocks)
    k_stage_fp32x2(const __grid_constant__ Grid g, const __grid_constant__ Layout L, const __grid_constant__ Ptr36 X,
                   PairBufs b, float* xn, const float* x2, const float* x3, PhysCoef<V> pc, StencilCoef<V> sc,
                   V h, V w6, Walk walk, StencilCoef<V> scl) {
    int ip, j, k;  // pair index along x
    if (!walk.site(g.nx >> 1, g.ny, g.nz, ip, j, k)) return;
    const int i0 = 2 * ip;
    using Acc = PairAcc<SrcPtr36<float>, COMP, V>;
    Acc A{{X}};
    A.place_ghost(i0, j, k, g.nx, L);
    A.s = sc;
    A.sl = scl;
    // L2 prefetch of this warp's lines of the epilogue operands (the RK4
    // accumulator and the state, read once each when the rates come out) and
    // of the stage input two planes up (read by the z stencils here and by
    // the blocks of the next planes).  The physics issues those loads late
    // and the warps wait on them.  Measured on GB300 at 256^3 with the 64x2
    // tile: 10.19 ms per step without, 9.75 with these prefetches; the stage
    // input at k+1 or k+3 instead of k+2: 9.80, at k+4: 9.91, two planes:
    // 10.02-10.15; the stage input alone (k+3): 9.96; the epilogue operands
    // alone: 3% slower than none.  Only full warps prefetch, the lines of
    // their lanes 0 and 16 (a warp's 64 sites where it lies in one row, its two
    // rows of 32 in tiles 16 wide): 72 lines of 128 bytes per buffer, two
    // or three per lane.  Plane k+2 <= nz+1 lies inside the ghosted box.
    // Only for 2^19 sites and more: ms per step without / with, 48^3 0.109 / 0.116,
    // 96^3 0.618 / 0.619, 128^3 1.300 / 1.285, 160^3 2.45 / 2.39, 256^3 9.70 / 9.37
    // (a smaller lattice has more of the lines in L2 already).  The compensated
    // mode, bound by its instructions, is faster without at every size: 64^3 0.314 /
    // 0.339, 128^3 1.77 / 1.88, 256^3 13.41 / 14.05.
    if (!COMP && g.S >= 1 << 19 && blockDim.x >= 16 && __activemask() == 0xffffffffu) {
        const int lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31;
        const int cl = __shfl_sync(0xffffffffu, A.c, 0), cu = __shfl_sync(0xffffffffu, A.c, 16);
        const int kz = 2 * L.px * L.py;
        for (int q = lane; q < 72; q += 32) {
            const bool upper = q & 1;
            const int64_t o = (q >> 1) * L.P + (upper ? cu : cl);
            if (STAGE > 1) {
                if (q >= 32) prefetch_l2(b.kacc + o);
                prefetch_l2(b.yhi + o);
            }
            if (STAGE == 4) {
                prefetch_l2(b.ylo + o);
                if (q >= 40) {
                    prefetch_l2(x2 + o);
                    prefetch_l2(x3 + o);
                }
            }
            prefetch_l2(reinterpret_cast<const float*>(X.p[q >> 1]) + (upper ? cu : cl) + kz);
        }
    }
    PairSink<STAGE, Acc> out{A, L, b, xn, h, w6, x2, x3};
    site_rates_fp32<V, BETA>(A, pc, out);
}

Ptr36 pack4(const void* base, int64_t S) {
    Ptr36 P;
    for (int a = 0; a < 36; ++a) P.p[a] = static_cast<const char*>(base) + (size_t)a * S * 4;
    return P;
}

template <bool BETA, int REG, bool COMP = false, class V = f2>
void step_pair(const Grid& g, const Layout& L, const Tiling& t, PairBufs b, float* xa, float* xb,
               const PhysCoef<V>& pc, const StencilCoef<V>& sc, const StencilCoef<V>& scl, double dt,
               cudaStream_t st) {
    dim3 gr, bl;
    const Walk walk = fp32_walk(g.nx / 2, g.ny, g.nz, t, true, gr, bl);
    const V h2((float)(dt / 2.)), h1((float)dt), w6((float)(dt / 6.)), z(0.f);
    float* x4m = b.kacc - 20 * L.P;  // X4's momenta
    Ptr36 X4 = pack4(xa, L.P);
    for (int a = 20; a < 36; ++a) X4.p[a] = x4m + a * L.P;
    const float* no = nullptr;
    k_stage_fp32x2<1, BETA, REG, COMP, V><<<gr, bl, 0, st>>>(g, L, pack4(b.yhi, L.P), b, xa, no, no, pc, sc, h2, w6, walk, scl);
    launch_ghost_fill_yz(g, L, xa, xa, st);
    k_stage_fp32x2<2, BETA, REG, COMP, V><<<gr, bl, 0, st>>>(g, L, pack4(xa, L.P), b, xb, no, no, pc, sc, h2, w6, walk, scl);
    launch_ghost_fill_yz(g, L, xb, xb, st);
    k_stage_fp32x2<3, BETA, REG, COMP, V><<<gr, bl, 0, st>>>(g, L, pack4(xb, L.P), b, xa, no, no, pc, sc, h1, w6, walk, scl);
    launch_ghost_fill_yz(g, L, xa, x4m, st);
    k_stage_fp32x2<4, BETA, REG, COMP, V><<<gr, bl, 0, st>>>(g, L, X4, b, nullptr, xa, xb, pc, sc, z, w6, walk, scl);
    launch_ghost_fill_yz(g, L, b.yhi, b.yhi, st);
}

template <bool BETA>
void step_pair_r(const Grid& g, const Layout& L, const Tiling& t, PairBufs b, float* xa, float* xb,
                 const PhysCoef<f2>& pc, const StencilCoef<f2>& sc, const StencilCoef<f2>& scl, bool comp,
                 double dt, cudaStream_t st) {
    if (comp)  // one register budget (<= 168) for the compensated mode
        step_pair<BETA, 2, true>(g, L, t, b, xa, xb, pc, sc, scl, dt, st);
    else if (t.reg == 1 && !t.pick)
        step_pair<BETA, 1>(g, L, t, b, xa, xb, pc, sc, scl, dt, st);
    else if (t.reg == 2 || t.pick)
        step_pair<BETA, 2>(g, L, t, b, xa, xb, pc, sc, scl, dt, st);
    else
        step_pair<BETA, 0>(g, L, t, b, xa, xb, pc, sc, scl, dt, st);
}

}  // namespace

cudaError_t launch_step_fp32_as_one(const Grid& g, const Layout& L, Fp32State y, Fp32Work w, const ewpt_params& p,
                                    double Jex, double gam, cudaStream_t st) {
    if (!fp32_as_one(g, p) || L.gx == 0) return cudaErrorInvalidValue;
    const StencilCoef<s2> sc = pair_stencil<s2>(make_stencil<float>(p.dx));
    step_pair<false, 2, false, s2>(g, L, kDefaultTiling, PairBufs{y.hi, y.lo, w.kacc}, w.xa, w.xb, make_phys<s2>(p, Jex, gam), sc, sc,
                        p.dt, st);
    return cudaGetLastError();
}

cudaError_t launch_step_fp32_pair(const Grid& g, const Layout& L, const Tiling& t, Fp32State y, Fp32Work w,
                                  const ewpt_params& p, double Jex, double gam, cudaStream_t st, bool comp) {
    if (g.nx % 2 != 0 || L.gx == 0) return cudaErrorInvalidValue;
    const PhysCoef<f2> pc = make_phys<f2>(p, Jex, gam);
    const StencilCoef<f2> sc = pair_stencil(make_stencil<float>(p.dx));
    const StencilCoef<f2> scl = pair_stencil_lo(make_stencil<double>(p.dx));
    PairBufs b{y.hi, y.lo, w.kacc};
    if (p.beta_w != 0.0 || p.beta_y != 0.0)
        step_pair_r<true>(g, L, t, b, w.xa, w.xb, pc, sc, scl, comp, p.dt, st);
    else
        step_pair_r<false>(g, L, t, b, w.xa, w.xb, pc, sc, scl, comp, p.dt, st);
    return cudaGetLastError();
}
