// stage.cu -- fused RK4 stage kernels of the FP32 form, one site per thread, and
// the conversions and ghost cells of its buffers.
//
// One launch = one stage of classical RK4 (gpu-kernels-rk4/main_rk4.jl:
// 6146-6437): the stage kernel rk4_step! (main_rk4.jl:52-661) with the
// reference's broadcast combination fused into its epilogue, so the 144
// broadcast kernels and ~72 temporary N^3 arrays of a reference step become
// four launches and no temporaries.  The stage input X is written once per
// stage by the previous launch; the periodic images along y and z lie in ghost
// cells, along x the neighbour offsets wrap.
//
// FP32 form (FP32 stencils and fluxes, compensated float hi/lo state):
//   stage 1:     kacc = k1;           X2 = y_hi + k1 dt/2
//   stage 2, 3:  kacc += 2 k_s;       X3 = y_hi + k2 dt/2,  X4 = y_hi + k3 dt
//   stage 4:     (y_hi, y_lo) += dt/6 (kacc + k4), compensated, in place
// (X_1 is y_hi itself; kacc of the fields is not stored, see Fp32Bufs).
// Bytes per site-update: 2480.  Bound by the latency of its loads (12 warps per
// SM; 128^3: issue slots 41% active, 3.5 TB/s).
#include <algorithm>

#include "accessors.cuh"
#include "physics_fp32.cuh"
#include "convert.cuh"

namespace {

// Register-budget variants of the stage kernels (launch bounds, blocks of at
// most 128 threads): 0 = registers at the compiler's choice (up to 255);
// 1 = at most 128 registers (4 blocks per SM); 2 = at most 168 registers (3
// blocks per SM).  The block shape (bx, by) is a launch parameter.
template <int REG>
struct RegBudget;
template <>
struct RegBudget<0> { static constexpr int kThreads = 128, kMinBlocks = 1; };
template <>
struct RegBudget<1> { static constexpr int kThreads = 128, kMinBlocks = 4; };
template <>
struct RegBudget<2> { static constexpr int kThreads = 128, kMinBlocks = 3; };

template <typename TL, typename T>
using GlobalAcc = SiteAcc<TL, T, SrcPtr36<TL>>;

// ------------------------------------------------------------- FP32 stage
// All five FP32 buffers use the ghosted layout L.  After each stage the
// ghost images of what it wrote (the next stage input, or the state high
// part after stage 4) are refreshed by k_ghost_fill_yz, so every stencil
// reads its neighbours with no wrap.
//
// The rate of a field (arrays 0-15) is its momentum, so k1, k2, k3 of a field
// are the momenta of the stage inputs y_hi, X2, X3 and no rate sum is stored
// for it: stage 4 forms k1 + 2 k2 + 2 k3 from them (the same roundings).  For
// that X2's momenta outlive stage 3, which writes X4's (arrays 20-35) into
// the unused arrays 0-15 of the rate sum instead of over X2's.  A step moves
// 2480 bytes per site instead of 2736.
struct Fp32Bufs {
    float* yhi;  // [36][P] state, high part (also the stage-1 stencil input)
    float* ylo;  // [36][P] state, low part
    float* kacc; // [36][P] arrays 16-35: rate sum k1, k1 + 2 k2, k1 + 2 k2 + 2 k3; 0-15: X4's momenta
};

template <int STAGE>
struct Fp32Sink {
    const GlobalAcc<float, float>& A;
    const Layout& L;
    Fp32Bufs b;
    float* xn;
    float h, w6;
    const float *x2, *x3;  // stage 4: the inputs of stages 2 and 3
    __device__ __forceinline__ void operator()(int a, float r) const {
        const int64_t q = a * L.P + A.c;
        if (STAGE < 4) {
            // kacc[q], yhi[q], ylo[q] are read and then written by this thread
            // only: the read-only path lets the loads issue ahead of stores
            if (a >= 16) b.kacc[q] = STAGE == 1 ? r : __ldg(b.kacc + q) + 2.f * r;
            float* x = STAGE == 3 && a >= 20 ? b.kacc - 20 * L.P : xn;  // X4's momenta
            x[q] = (STAGE == 1 ? A.v(a) : __ldg(b.yhi + q)) + h * r;    // X1 == y_hi
        } else {
            float k;
            if (a < 16) {
                const int64_t m = q + 20 * L.P;
                k = __ldg(b.yhi + m) + 2.f * __ldg(x2 + m);
                k = k + 2.f * __ldg(x3 + m);
            } else {
                k = __ldg(b.kacc + q);
            }
            const float s = k + r;
            float hi = __ldg(b.yhi + q), lo = __ldg(b.ylo + q);
            acc_hilo(hi, lo, w6 * s);
            b.yhi[q] = hi;
            b.ylo[q] = lo;
        }
    }
};

template <int STAGE, bool BETA, int REG>
__global__ void __launch_bounds__(RegBudget<REG>::kThreads, RegBudget<REG>::kMinBlocks)
    k_stage_fp32(const __grid_constant__ Grid g, const __grid_constant__ Layout L, const __grid_constant__ Ptr36 X,
                 Fp32Bufs b, float* xn, const float* x2, const float* x3, PhysCoef<float> pc, StencilCoef<float> sc,
                 float h, float w6, Walk walk) {
    int i, j, k;
    if (!walk.site(g.nx, g.ny, g.nz, i, j, k)) return;
    GlobalAcc<float, float> A{{X}};
    A.place_ghost(i, j, k, g.nx, L);
    A.s = sc;
    Fp32Sink<STAGE> out{A, L, b, xn, h, w6, x2, x3};
    site_rates_fp32<float, BETA>(A, pc, out);
}

// FP64 arrays <-> (hi, lo) in layout L (ghost cells left to k_ghost_fill).
// One block per piece of a plane (a*nz + k over the 36 arrays); a thread walks
// its piece in steps of the block, carrying (i, j) without a division.
// Bound by memory: at 256^3 split / join move 9.7 GB and took 5.12 / 4.48 ms
// with a 64-bit division pair and C casts per value (the FP64 pipe,
// convert.cuh).
constexpr int kConvThreads = 256, kConvPiece = 16 * kConvThreads;

template <class F>
__device__ __forceinline__ void conv_walk(const Grid& g, F f) {
    const int A = g.nx * g.ny, pieces = (A + kConvPiece - 1) / kConvPiece;
    const int plane = blockIdx.x / pieces, a = plane / g.nz, k = plane - a * g.nz;
    const int q0 = (blockIdx.x - plane * pieces) * kConvPiece, q1 = min(A, q0 + kConvPiece);
    int q = q0 + (int)threadIdx.x;
    int j = q / g.nx, i = q - j * g.nx;
    const int dj = kConvThreads / g.nx, di = kConvThreads - dj * g.nx;
    const int64_t base = (int64_t)k * A;
#pragma unroll 4
    for (; q < q1; q += kConvThreads) {
        f(a, base + q, i, j, k);
        i += di;
        j += dj;
        if (i >= g.nx) {
            i -= g.nx;
            ++j;
        }
    }
}

__global__ void __launch_bounds__(kConvThreads) k_split(Grid g, Layout L, const __grid_constant__ Ptr36 src,
                                                        float* __restrict__ hi, float* __restrict__ lo) {
    conv_walk(g, [&](int a, int64_t c, int i, int j, int k) {
        const int64_t d = a * L.P + L.at(i, j, k);
        split_f64(__ldg(reinterpret_cast<const double*>(src.p[a]) + c), hi[d], lo[d]);
    });
}

__global__ void __launch_bounds__(kConvThreads) k_join(Grid g, Layout L, const float* __restrict__ hi,
                                                       const float* __restrict__ lo,
                                                       const __grid_constant__ MPtr36 dst) {
    conv_walk(g, [&](int a, int64_t c, int i, int j, int k) {
        const int64_t d = a * L.P + L.at(i, j, k);
        reinterpret_cast<double*>(dst.p[a])[c] = join_f64(__ldg(hi + d), __ldg(lo + d));
    });
}

// Ghost images of a ghosted buffer, one warp per work item over a grid of a
// few blocks per SM: first the y- and z-face rows (a warp copies one row of
// nx sites into one of the 3 + 3 ghost rows of an x-y plane, or into a row
// of one of the 3 + 3 ghost planes), then the x faces (a warp serves 4 rows,
// 8 cells each: the 4 ghost cells before the row and the 4 after it).  The x
// faces cost most of the time (16-byte pieces of every row, 0.86 GB of DRAM
// reads per launch at 256^3), so only the TMA-staged kernel, whose boxes read
// them, has them filled; the other FP32 kernels wrap x in their neighbour
// offsets and take k_ghost_fill_yz.  Every
// cell copies the site it is the periodic image of; the box edges and
// corners are left alone (no axis-aligned stencil reaches them).
__global__ void __launch_bounds__(256) k_ghost_fill(Grid g, Layout L, float* __restrict__ buf) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int px = L.px, pxy = L.px * L.py;
    const int lane = threadIdx.x & 31;
    const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const int per_a = 6 * (ny + nz);
    for (int r = w0; r < 36 * per_a; r += nw) {
        const int a = r / per_a, e = r - a * per_a;
        float* arr = buf + a * L.P + L.o0;  // site (0, 0, 0)
        int doff, soff;
        if (e < 6 * nz) {
            const int yg = e % 6, k = e / 6;
            doff = (yg < 3 ? yg - 3 : ny + yg - 3) * px + k * pxy;
            soff = (yg < 3 ? ny + yg - 3 : yg - 3) * px + k * pxy;
        } else {
            const int zg = (e - 6 * nz) % 6, j = (e - 6 * nz) / 6;
            doff = j * px + (zg < 3 ? zg - 3 : nz + zg - 3) * pxy;
            soff = j * px + (zg < 3 ? nz + zg - 3 : zg - 3) * pxy;
        }
        for (int i = lane; i < nx; i += 32) arr[doff + i] = arr[soff + i];
    }
    const int rows = ny * nz, quads = (36 * rows + 3) / 4;
    const int xg = lane & 7;
    const int di = xg < 4 ? xg - 4 : nx + xg - 4, si = xg < 4 ? nx + xg - 4 : xg - 4;
    for (int q = w0; q < quads; q += nw) {
        const int rr = 4 * q + (lane >> 3);
        if (rr >= 36 * rows) continue;
        const int a = rr / rows, row = rr - a * rows;
        float* base = buf + a * L.P + L.o0 + (row % ny) * px + (row / ny) * pxy;
        base[di] = base[si];
    }
}

// The same without the x faces, and only the arrays some stencil reads along
// the face's axis: the 20 fields and, along y or z, the gauge momentum of that
// component (the Gauss-law divergence).  One row per warp.  Array a lies at
// fld + a*P for a < 20, at mom + a*P from 20 on.
__global__ void __launch_bounds__(256) k_ghost_fill_yz(Grid g, Layout L, float* __restrict__ fld,
                                                       float* __restrict__ mom) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int px = L.px, pxy = L.px * L.py;
    const int lane = threadIdx.x & 31;
    int r = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int per_a = 6 * (ny + nz);
    if (r >= 24 * per_a) return;
    const int q = r / per_a;
    r -= q * per_a;
    const bool yface = r < 6 * nz;
    if (!yface) r -= 6 * nz;
    const int gh = r % 6, line = r / 6;
    const int a = q < 20 ? q : 20 + 3 * (q - 19) + (yface ? 2 : 3);
    float* arr = (a < 20 ? fld : mom) + a * L.P + L.o0;  // site (0, 0, 0)
    const int n = yface ? ny : nz, step = yface ? px : pxy, base = line * (yface ? pxy : px);
    const int doff = base + (gh < 3 ? gh - 3 : n + gh - 3) * step;
    const int soff = base + (gh < 3 ? n + gh - 3 : gh - 3) * step;
#pragma unroll 4
    for (int i = lane; i < nx; i += 32) arr[doff + i] = arr[soff + i];
}

Ptr36 pack(const void* base, int64_t S, size_t elem) {
    Ptr36 P;
    for (int a = 0; a < 36; ++a) P.p[a] = static_cast<const char*>(base) + (size_t)a * S * elem;
    return P;
}

}  // namespace

int tiling_max_threads(int reg) { return reg >= 0 && reg <= 2 ? 128 : 0; }

// FP32 form: stage inputs ping-pong between xa and xb.
template <bool BETA, int REG>
static void step_fp32(const Grid& g, const Layout& L, const Tiling& t, Fp32Bufs b, float* xa, float* xb,
                      const PhysCoef<float>& pc, const StencilCoef<float>& sc, double dt, cudaStream_t st) {
    dim3 gr, bl;
    const Walk walk = fp32_walk(g.nx, g.ny, g.nz, t, false, gr, bl);
    const float h2 = (float)(dt / 2.), h1 = (float)dt, w6 = (float)(dt / 6.);
    float* x4m = b.kacc - 20 * L.P;  // X4's momenta
    Ptr36 X4 = pack(xa, L.P, 4);
    for (int a = 20; a < 36; ++a) X4.p[a] = x4m + a * L.P;
    const float* no = nullptr;
    k_stage_fp32<1, BETA, REG><<<gr, bl, 0, st>>>(g, L, pack(b.yhi, L.P, 4), b, xa, no, no, pc, sc, h2, w6, walk);
    launch_ghost_fill_yz(g, L, xa, xa, st);
    k_stage_fp32<2, BETA, REG><<<gr, bl, 0, st>>>(g, L, pack(xa, L.P, 4), b, xb, no, no, pc, sc, h2, w6, walk);
    launch_ghost_fill_yz(g, L, xb, xb, st);
    k_stage_fp32<3, BETA, REG><<<gr, bl, 0, st>>>(g, L, pack(xb, L.P, 4), b, xa, no, no, pc, sc, h1, w6, walk);
    launch_ghost_fill_yz(g, L, xa, x4m, st);
    k_stage_fp32<4, BETA, REG><<<gr, bl, 0, st>>>(g, L, X4, b, nullptr, xa, xb, pc, sc, 0.f, w6, walk);
    launch_ghost_fill_yz(g, L, b.yhi, b.yhi, st);
}

template <bool BETA>
static void step_fp32_r(const Grid& g, const Layout& L, const Tiling& t, Fp32Bufs b, float* xa, float* xb,
                        const PhysCoef<float>& pc, const StencilCoef<float>& sc, double dt, cudaStream_t st) {
    // picked: <= 168 registers, or the compiler's choice (8 warps per SM) where the
    // lattice has no more sites than 7 warps per SM (16^3 0.049 against
    // 0.053 ms per step, 24^3 0.051 against 0.057, 32^3 0.056 against 0.059; 33^3
    // 0.081 against 0.076, 36^3 0.093 against 0.080)
    const int reg = !t.pick ? t.reg : g.S > 152 * 7 * 32 ? 2 : 0;
    if (reg == 1)
        step_fp32<BETA, 1>(g, L, t, b, xa, xb, pc, sc, dt, st);
    else if (reg == 2)
        step_fp32<BETA, 2>(g, L, t, b, xa, xb, pc, sc, dt, st);
    else
        step_fp32<BETA, 0>(g, L, t, b, xa, xb, pc, sc, dt, st);
}

cudaError_t launch_step_fp32(const Grid& g, const Layout& L, const Tiling& t, Fp32State y, Fp32Work w,
                             const ewpt_params& p, double Jex, double gam, cudaStream_t st) {
    if (L.gx == 0) return cudaErrorInvalidValue;  // the single-lattice kernels read ghost cells
    if (t.pick && fp32_as_one(g, p)) return launch_step_fp32_as_one(g, L, y, w, p, Jex, gam, st);
    const PhysCoef<float> pc = make_phys<float>(p, Jex, gam);
    const StencilCoef<float> sc = make_stencil<float>(p.dx);
    Fp32Bufs b{y.hi, y.lo, w.kacc};
    if (p.beta_w != 0.0 || p.beta_y != 0.0)
        step_fp32_r<true>(g, L, t, b, w.xa, w.xb, pc, sc, p.dt, st);
    else
        step_fp32_r<false>(g, L, t, b, w.xa, w.xb, pc, sc, p.dt, st);
    return cudaGetLastError();
}

cudaError_t launch_ghost_fill(const Grid& g, const Layout& L, float* buf, cudaStream_t st, bool xfaces) {
    if (L.gx == 0) return cudaSuccess;
    if (!xfaces) return launch_ghost_fill_yz(g, L, buf, buf, st);
    k_ghost_fill<<<152 * 8, 256, 0, st>>>(g, L, buf);
    return cudaGetLastError();
}

cudaError_t launch_ghost_fill_yz(const Grid& g, const Layout& L, float* fld, float* mom, cudaStream_t st) {
    const int64_t rows = (int64_t)24 * 6 * (g.ny + g.nz);
    k_ghost_fill_yz<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(g, L, fld, mom);
    return cudaGetLastError();
}

static unsigned conv_grid(const Grid& g, int arrays) {
    return (unsigned)((g.nx * g.ny + kConvPiece - 1) / kConvPiece) * (unsigned)arrays * (unsigned)g.nz;
}

cudaError_t launch_fp32_split(const Grid& g, const Layout& L, const Ptr36& src, Fp32State dst, cudaStream_t st,
                              bool xfaces) {
    k_split<<<conv_grid(g, 36), kConvThreads, 0, st>>>(g, L, src, dst.hi, dst.lo);
    return launch_ghost_fill(g, L, dst.hi, st, xfaces);
}

cudaError_t launch_fp32_join(const Grid& g, const Layout& L, Fp32State src, const MPtr36& dst, cudaStream_t st,
                             int arrays) {
    k_join<<<conv_grid(g, arrays), kConvThreads, 0, st>>>(g, L, src.hi, src.lo, dst);
    return cudaGetLastError();
}
