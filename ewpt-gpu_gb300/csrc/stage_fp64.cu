// stage_fp64.cu -- the FP64 form's RK4 stages and the drop-in rates, 6th order:
// four warps evolve 32 sites together.
//
// One launch = one stage of classical RK4 (gpu-kernels-rk4/main_rk4.jl:
// 6146-6437), as in stage.cu: rk4_step! (main_rk4.jl:52-661) with the
// reference's broadcast combination in the epilogue, in the reference's
// accumulation order:
//   stage 1: k = f(y);   yn = y  + k dt/6;  X2 = y + k dt/2
//   stage 2: k = f(X2);  yn = yn + k dt/3;  X3 = y + k dt/2
//   stage 3: k = f(X3);  yn = yn + k dt/3;  X4 = y + k dt
//   stage 4: k = f(X4);  y  = yn + k dt/6
//
// A block of 128 threads owns 32 sites, lane = site.  First each warp takes a
// quarter of the stencils (four gradients with Laplacian, a gradient, a
// divergence; integer arithmetic, fixstencil.cuh) and leaves them in shared
// memory, 80 doubles per site.  Then warp 1 + a evaluates colour a -- W^a_i,
// Gamma^a and one component of Y -- and the covariant Higgs derivatives along
// axis a, and warp 0 the momentum rates, the local Higgs terms and Sigma, with
// the axes' parts added when they are there: some 100 and 120 FP64 instructions.
// The equations are those of physics.cuh.
//
// Bound by the FP64 pipe (one warp instruction per 64 cycles and SM quarter):
// 487 FP64 instructions per 32 sites and stage, the pipe 81-83% busy at 96^3 (ncu;
// chains of independent FMAs reach 84%; shared-memory latency and instruction
// fetch the largest stalls).  A site per
// thread took 128-255 registers through ~15 k instructions: 16 warps per SM ran
// the pipe at 66%, and a lattice of less than a warp per SM quarter ran at the
// latency of that one chain.  Four warps of 72 registers, 28 per SM, one such
// chain a quarter as long.  Step at one site per thread -> four warps: 24 x 20 x
// 28 0.171 -> 0.0985 ms, 64^3 1.20 -> 1.12, 75 x 61 x 90 1.84 -> 1.72, 128^3 9.29
// -> 8.40, 256^3 76.2 -> 66.8 (532 FP64 instructions); with the units of the
// momentum rates in the sink's weights, negations folded and no division
// without damping (487) 64^3 1.01, 128^3 7.58, 256^3 60.2; with stencils that are
// odd to the bit and an exponent per line (fixstencil.cuh) 24 x 20 x 28 0.097,
// 64^3 1.04, 75 x 61 x 90 1.59, 128^3 7.83, 256^3 62.0.  The Higgs part in one warp instead of split by
// axis: 0.117 and 1.23 at 24 x 20 x 28 and 64^3.  The stencils out of line, with
// the neighbours' offsets in local memory: 0.107 and 1.15.  Blocks per SM, six,
// seven, eight: 24 x 20 x 28 0.098, 0.0985, 0.105; 256^3 68.8, 66.8, 66.0.
#include "stage_fp64.cuh"

namespace {

// sites: how many, from plane g.k0 on, x fastest
template <int STAGE, bool BETA, class Out>
__device__ __forceinline__ void evolve(const Grid& g, const Ptr36& X, const Coef& pc, int sites, const Out& out) {
    __shared__ SharedOf<BETA> sh;
    // The roles turn with the block: warp w of every block runs on SM quarter
    // w % 4, and a colour has a little more to do than the Higgs warp.
    const int lane = threadIdx.x & 31, warp = ((threadIdx.x >> 5) + blockIdx.x) & (kWarps - 1);
    const int64_t q0 = (int64_t)blockIdx.x * kSites + lane;
    const bool live = q0 < sites;
    const int q = live ? (int)q0 : sites - 1;  // lanes past the end repeat the last site and write nothing
    const int row = q / g.nx, i = q - row * g.nx, pl = row / g.ny, j = row - pl * g.ny;
    FixAcc A{X, g};
    A.place(i, j, pl + g.k0);
    stencils(A, sh, lane, warp);
    __syncthreads();
    if (warp == 0)
        higgs_warp<STAGE, BETA>(A, pc, sh, lane, live, out);
    else
        colour_warp<STAGE, BETA>(A, pc, sh, lane, live, warp - 1, out);
}

template <int STAGE, bool BETA>
__global__ void __launch_bounds__(kSites* kWarps, 7)
    k_stage_fp64(Grid g, const __grid_constant__ Ptr36 X, const __grid_constant__ StageSink out,
                 const __grid_constant__ Coef pc, int sites) {
    evolve<STAGE, BETA>(g, X, pc, sites, out);
}

template <bool BETA>
__global__ void __launch_bounds__(kSites* kWarps, 7)
    k_rates_fp64(Grid g, const __grid_constant__ Ptr36 X, const __grid_constant__ RatesOut out,
                 const __grid_constant__ Coef pc, int sites) {
    evolve<0, BETA>(g, X, pc, sites, out);
}

unsigned blocks_for(int64_t sites) { return (unsigned)((sites + kSites - 1) / kSites); }

// stage s over `sites` sites from plane g.k0 on
template <bool BETA>
void stage_fp64(const Grid& g, int stage, double* y, double* yn, double* xa, double* xb, const Coef& pc,
                double dt, int sites, cudaStream_t st) {
    const unsigned nb = blocks_for(sites);
    const int nt = kSites * kWarps;
    auto sink = [&](double* xn, double w, double h) {
        return StageSink{y, yn, xn, g.S, {w, w * pc.hgw_o, w * pc.gw_o}, {h, h * pc.hgw_o, h * pc.gw_o}};
    };
    auto in = [&](const double* x) { return arrays36(x, g.S); };
    switch (stage) {
        case 1: k_stage_fp64<1, BETA><<<nb, nt, 0, st>>>(g, in(y), sink(xa, dt / 6., dt / 2.), pc, sites); break;
        case 2: k_stage_fp64<2, BETA><<<nb, nt, 0, st>>>(g, in(xa), sink(xb, dt / 3., dt / 2.), pc, sites); break;
        case 3: k_stage_fp64<3, BETA><<<nb, nt, 0, st>>>(g, in(xb), sink(xa, dt / 3., dt), pc, sites); break;
        default: k_stage_fp64<4, BETA><<<nb, nt, 0, st>>>(g, in(xa), sink(y, dt / 6., 0.0), pc, sites);
    }
}

}  // namespace

cudaError_t launch_rates_fp64(const Grid& g, const Ptr36& in, const MPtr36& out, const ewpt_params& p, double Jex,
                              double gam, cudaStream_t st) {
    const Coef pc = make_coef(p, Jex, gam);
    const RatesOut o{out, {1.0, pc.hgw_o, pc.gw_o}};
    const int sites = (int)((int64_t)g.nx * g.ny * g.nz);
    if (p.beta_w != 0.0 || p.beta_y != 0.0)
        k_rates_fp64<true><<<blocks_for(sites), kSites * kWarps, 0, st>>>(g, in, o, pc, sites);
    else
        k_rates_fp64<false><<<blocks_for(sites), kSites * kWarps, 0, st>>>(g, in, o, pc, sites);
    return cudaGetLastError();
}

cudaError_t launch_stage_fp64_planes(const Grid& g, int stage, int k0, int k1, double* y, double* yn, double* xa,
                                     double* xb, const ewpt_params& p, double Jex, double gam, cudaStream_t st) {
    if (k0 < 0 || k1 > g.nz || k0 >= k1) return k0 == k1 ? cudaSuccess : cudaErrorInvalidValue;
    const Coef pc = make_coef(p, Jex, gam);
    Grid gw = g;
    gw.k0 = k0;
    const int sites = (int)((int64_t)g.nx * g.ny * (k1 - k0));
    if (p.beta_w != 0.0 || p.beta_y != 0.0)
        stage_fp64<true>(gw, stage, y, yn, xa, xb, pc, p.dt, sites, st);
    else
        stage_fp64<false>(gw, stage, y, yn, xa, xb, pc, p.dt, sites, st);
    return cudaGetLastError();
}

cudaError_t launch_stage_fp64(const Grid& g, int stage, double* y, double* yn, double* xa, double* xb,
                              const ewpt_params& p, double Jex, double gam, cudaStream_t st) {
    return launch_stage_fp64_planes(g, stage, 0, g.nz, y, yn, xa, xb, p, Jex, gam, st);
}

cudaError_t launch_step_fp64(const Grid& g, double* y, double* yn, double* xa, double* xb, const ewpt_params& p,
                             double Jex, double gam, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (int stage = 1; stage <= 4 && e == cudaSuccess; ++stage)
        e = launch_stage_fp64(g, stage, y, yn, xa, xb, p, Jex, gam, st);
    return e;
}
