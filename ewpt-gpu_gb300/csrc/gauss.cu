// gauss.cu -- projection of an FP64 state's electric fields onto the
// discrete Gauss law, on the device.
//
// The Gauss constraints of the evolution are the gp2 parts of k_Gamma and
// k_Sigma (main_rk4.jl:603-655): d_i E^a_i = rho^a with
//   rho^a = g (Higgs charge  phi^T M_a pi  -  sum_i (W^b_i E^c_i - W^c_i E^b_i))
// for (a, b, c) cyclic, and d_i E^Y_i = rho_Y = g' phi^T M_Y pi, where E are
// the gauge momenta, pi the Higgs momenta and d_i the 6th-order central
// difference.  A thermal state draws E and pi freely; one projection
// iteration makes it satisfy the constraints:
//   1. neutralise: the central-difference divergence cannot produce the zero
//      mode or the staggered modes (-1)^(e.x) (e_i = 1 only on even axes), so
//      the charges must have no component there.  The Higgs momenta move
//      along the charge generators, pi += sum_b c_b(x) M_b^T phi with c_b
//      constant on each of the 8 parity classes of the sites; the 4 x ne
//      coefficients solve a least-squares system whose entries are
//      parity-class moments of rho and of phi^T M_a M_b^T phi (one reduction
//      kernel, then a one-sided Jacobi SVD of the <= 32 x 32 system on the
//      host, the minimum-norm solution as numpy's lstsq gives it);
//   2. project: per group (the three SU(2) colours and U(1)), with rho taken
//      before the iteration, E <- E - grad chi with d.d chi = d.E - rho: the
//      divergence and the gradient are the stencils, and chi comes from one
//      forward and one backward real FFT of the source with the squared symbol
//      s(theta) = (90 sin theta - 18 sin 2 theta + 2 sin 3 theta) / (60 dx)
//      (cuFFT D2Z / Z2D); modes with |s|^2 <= 1e-12 max |s|^2 are left alone.
// The rho^a of the next iteration sees the projected E (the SU(2) charge
// depends on E), so the residual falls by iterations.  ewpt/ic.py
// gauss_project does the same steps on the host, with step 2 wholly in Fourier
// space (E and rho transformed, E transformed back).
//
// Bound by the FP64 pipe: the FFTs (96^3: 0.11 ms each, 8 per iteration; 28
// when E itself is transformed), then the charges.  20 iterations at 96^3 on
// a thermal state took 110 ms with 28 FFTs, the symbol's nine sines per mode
// and the moments in shared-memory atomics.
#include <cufft.h>

#include <cmath>
#include <string>
#include <vector>

#include "ewpt_ctx.cuh"
#include "fixstencil.cuh"

namespace {

constexpr int kNQ = 20;  // moments per parity class: 4 charges, then 16 generator overlaps
// what the device sums of them: the 4 charges, |phi|^2 and the overlaps of the
// SU(2) generators with the U(1) generator.  The SU(2) generators turn phi into
// three orthogonal vectors of its length, so the other overlaps are |phi|^2 or 0.
constexpr int kND = 8;

// u = M_b^T phi of the charge generators M_b (b = 0, 1, 2: SU(2); 3: U(1))
__device__ __forceinline__ void gen_t(int b, const double* ph, double* u) {
    switch (b) {
        case 0: u[0] = -ph[3], u[1] = ph[2], u[2] = -ph[1], u[3] = ph[0]; break;
        case 1: u[0] = ph[2], u[1] = ph[3], u[2] = -ph[0], u[3] = -ph[1]; break;
        case 2: u[0] = -ph[1], u[1] = ph[0], u[2] = ph[3], u[3] = -ph[2]; break;
        default: u[0] = -ph[1], u[1] = ph[0], u[2] = -ph[3], u[3] = ph[2];
    }
}

// rho^1..3 and rho_Y at site c of an FP64 [36][S] state with Higgs field ph
// and momentum pi
__device__ __forceinline__ void site_charges(const double* __restrict__ y, int64_t S, int64_t c, const double* ph,
                                             const double* pi, double gw, double gy, double* rho) {
    double u[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        gen_t(a, ph, u);  // phi^T M_a pi = (M_a^T phi) . pi
        double h = u[0] * pi[0] + u[1] * pi[1] + u[2] * pi[2] + u[3] * pi[3];
        if (a < 3) {
            const int b = (a + 1) % 3, cc = (a + 2) % 3;
#pragma unroll
            for (int i = 0; i < 3; ++i)
                h -= y[(4 + 3 * b + i) * S + c] * y[(24 + 3 * cc + i) * S + c] -
                     y[(4 + 3 * cc + i) * S + c] * y[(24 + 3 * b + i) * S + c];
            rho[a] = gw * h;
        } else {
            rho[a] = gy * h;
        }
    }
}

constexpr int kMomentBlocks = 4 * 152, kMomentWarps = 8;

// Sums over each parity class of the kND quantities.  Block b takes the rows
// whose (j, k) have the parities of b % 4, a warp a row at a time, a lane the
// sites of its own parity, so every thread sums one class in registers.
// part[block][parity of i][kND].
__global__ void __launch_bounds__(32 * kMomentWarps) k_class_moments(Grid g, const double* __restrict__ y, double gw,
                                                                     double gy, double* __restrict__ part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pj = blockIdx.x & 1, pk = (blockIdx.x >> 1) & 1;
    const int nj = (g.ny + 1 - pj) / 2, nk = (g.nz + 1 - pk) / 2;
    double s[kND] = {};
    for (int r = (blockIdx.x >> 2) * kMomentWarps + warp; r < nj * nk; r += (kMomentBlocks / 4) * kMomentWarps) {
        const int j = 2 * (r % nj) + pj, k = 2 * (r / nj) + pk;
        const int64_t row = (int64_t)g.nx * (j + (int64_t)g.ny * k);
        for (int i = lane; i < g.nx; i += 32) {
            const int64_t q = row + i;
            double rho[4], ph[4], pi[4], uy[4], u[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                ph[a] = y[a * g.S + q];
                pi[a] = y[(20 + a) * g.S + q];
            }
            site_charges(y, g.S, q, ph, pi, gw, gy, rho);
            gen_t(3, ph, uy);
#pragma unroll
            for (int a = 0; a < 4; ++a) s[a] += rho[a];
            s[4] += ph[0] * ph[0] + ph[1] * ph[1] + ph[2] * ph[2] + ph[3] * ph[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                gen_t(a, ph, u);
                s[5 + a] += u[0] * uy[0] + u[1] * uy[1] + u[2] * uy[2] + u[3] * uy[3];
            }
        }
    }
    __shared__ double sh[kMomentWarps][2][kND];
#pragma unroll
    for (int t = 0; t < kND; ++t) {
        for (int off = 16; off > 1; off >>= 1) s[t] += __shfl_down_sync(0xffffffffu, s[t], off);
        if (lane < 2) sh[warp][lane][t] = s[t];
    }
    __syncthreads();
    if (threadIdx.x < 2 * kND) {
        double v = 0.0;
        for (int w = 0; w < kMomentWarps; ++w) v += (&sh[w][0][0])[threadIdx.x];
        part[blockIdx.x * 2 * kND + threadIdx.x] = v;
    }
}

// out[class][kND]: one warp per sum
__global__ void __launch_bounds__(1024) k_fold_moments(const double* __restrict__ part, double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < 8 * kND; q += 32) {
        const int cls = q / kND, t = q % kND;  // class = pk*4 + pj*2 + pi
        double v = 0.0;
        for (int b = (cls >> 1) + 4 * lane; b < kMomentBlocks; b += 128) v += part[b * 2 * kND + (cls & 1) * kND + t];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) out[q] = v;
    }
}

// difference operator over a [.][S] buffer at the site of this thread
__device__ __forceinline__ bool site_of(const Grid& g, const double* y, FixDiff& A, int* parity) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if ((int64_t)blockIdx.x * blockDim.x + threadIdx.x >= g.S) return false;
    const int row = q / g.nx, i = q - row * g.nx, k = row / g.ny, j = row - k * g.ny;
    A.y = y;
    A.S = g.S;
    A.c = q;
    axis_offsets(i, g.nx, 1, A.o[0]);
    axis_offsets(j, g.ny, g.nx, A.o[1]);
    axis_offsets(k, g.nz, g.nx * g.ny, A.o[2]);
    if (parity) *parity = (k & 1) * 4 + (j & 1) * 2 + (i & 1);
    return true;
}

struct Table32 {
    double t[32];
};

// pi += table[b][class(x)] M_b^T phi, then src[a] = d_i E^a_i - rho^a
__global__ void __launch_bounds__(128, 4) k_source(Grid g, double* __restrict__ y, const __grid_constant__ Table32 tab,
                                                   double gw, double gy, double t, double* __restrict__ src, int64_t Sp) {
    FixDiff A;
    int cls;
    if (!site_of(g, y, A, &cls)) return;
    const int64_t q = A.c;
    double ph[4], pi[4], u[4], rho[4], d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int a = 0; a < 4; ++a) ph[a] = y[a * g.S + q];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        gen_t(b, ph, u);
        const double w = tab.t[b * 8 + cls];
#pragma unroll
        for (int a = 0; a < 4; ++a) d[a] += w * u[a];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        pi[a] = y[(20 + a) * g.S + q] + d[a];
        y[(20 + a) * g.S + q] = pi[a];
    }
    site_charges(y, g.S, q, ph, pi, gw, gy, rho);
#pragma unroll
    for (int a = 0; a < 4; ++a) src[a * Sp + q] = t * A.div(24 + 3 * a) - rho[a];
}

// half spectrum (x: 0..nx/2) of the source -> of chi: times -1 / (S |s|^2),
// zero where |s|^2 <= cut; the tables hold each axis' s^2
__global__ void __launch_bounds__(256) k_solve(Grid g, const double* __restrict__ sx, const double* __restrict__ sy,
                                               const double* __restrict__ sz, double cut,
                                               cufftDoubleComplex* __restrict__ C) {
    const int hx = g.nx / 2 + 1;
    const int64_t H = (int64_t)hx * g.ny * g.nz;
    const double inv = 1.0 / (double)g.S;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < H; q += (int64_t)gridDim.x * blockDim.x) {
        const int row = (int)(q / hx), i = (int)(q - (int64_t)row * hx), k = row / g.ny, j = row - k * g.ny;
        const double s2 = sx[i] + sy[j] + sz[k];
        const double f = s2 > cut ? -inv / s2 : 0.0;
        const cufftDoubleComplex v = C[q];
        C[q] = make_cuDoubleComplex(f * v.x, f * v.y);
    }
}

// E^a_i -= d_i chi^a
__global__ void __launch_bounds__(128, 4) k_subtract(Grid g, double* __restrict__ y, const double* __restrict__ chi,
                                                     int64_t Sp, double t) {
    FixDiff A;
    if (!site_of(g, chi, A, nullptr)) return;
    A.S = Sp;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        double d[3];
        A.grad(a, d[0], d[1], d[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            double* e = y + (24 + 3 * a + i) * g.S + A.c;
            *e = fma(-t, d[i], *e);
        }
    }
}

double host_symbol(double th, double dx) {
    return (90.0 * std::sin(th) - 18.0 * std::sin(2.0 * th) + 2.0 * std::sin(3.0 * th)) / (60.0 * dx);
}

// The staggered vectors e = (ez, ey, ex), e_i = 1 only on even axes, ez outermost.
std::vector<int> null_vectors(const Grid& g) {
    std::vector<int> es;
    for (int ez = 0; ez < (g.nz % 2 == 0 ? 2 : 1); ++ez)
        for (int ey = 0; ey < (g.ny % 2 == 0 ? 2 : 1); ++ey)
            for (int ex = 0; ex < (g.nx % 2 == 0 ? 2 : 1); ++ex) es.push_back(ez * 4 + ey * 2 + ex);
    return es;
}

// sum_x (-1)^(e.x) f(x) from the parity-class sums s[class] (class = pz*4 + py*2 + px)
double moment(const double* s, int stride, int e) {
    double m = 0.0;
    for (int c = 0; c < 8; ++c) m += (__builtin_popcount(c & e) & 1 ? -1.0 : 1.0) * s[c * stride];
    return m;
}

// Minimum-norm least-squares solution of A x = b (m x n, row-major), by a
// one-sided Jacobi SVD (Hestenes); singular values below
// eps * max(m, n) * sigma_max are dropped, as numpy's lstsq does by default.
std::vector<double> lstsq(const std::vector<double>& rows, int m, int n, const std::vector<double>& b) {
    // columns of A and V back to back: the rotations run over whole columns
    std::vector<double> A((size_t)n * m), V((size_t)n * n, 0.0);
    for (int i = 0; i < m; ++i)
        for (int j = 0; j < n; ++j) A[(size_t)j * m + i] = rows[(size_t)i * n + j];
    for (int i = 0; i < n; ++i) V[(size_t)i * n + i] = 1.0;
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0;
        for (int p = 0; p < n - 1; ++p)
            for (int q = p + 1; q < n; ++q) {
                double al = 0.0, be = 0.0, ga = 0.0;
                double *ap = &A[(size_t)p * m], *aq = &A[(size_t)q * m], *vp = &V[(size_t)p * n], *vq = &V[(size_t)q * n];
                for (int i = 0; i < m; ++i) {
                    const double x = ap[i], y = aq[i];
                    al += x * x;
                    be += y * y;
                    ga += x * y;
                }
                if (ga == 0.0 || std::fabs(ga) <= 1e-15 * std::sqrt(al * be)) continue;
                off = std::fmax(off, std::fabs(ga) / std::sqrt(al * be));
                const double zeta = (be - al) / (2.0 * ga);
                const double t = (zeta >= 0 ? 1.0 : -1.0) / (std::fabs(zeta) + std::sqrt(1.0 + zeta * zeta));
                const double c = 1.0 / std::sqrt(1.0 + t * t), s = c * t;
                for (int i = 0; i < m; ++i) {
                    const double x = ap[i], y = aq[i];
                    ap[i] = c * x - s * y;
                    aq[i] = s * x + c * y;
                }
                for (int i = 0; i < n; ++i) {
                    const double x = vp[i], y = vq[i];
                    vp[i] = c * x - s * y;
                    vq[i] = s * x + c * y;
                }
            }
        if (off < 1e-15) break;
    }
    std::vector<double> sig(n), x(n, 0.0);
    double smax = 0.0;
    for (int k = 0; k < n; ++k) {
        double s = 0.0;
        for (int i = 0; i < m; ++i) s += A[(size_t)k * m + i] * A[(size_t)k * m + i];
        sig[k] = std::sqrt(s);
        smax = std::fmax(smax, sig[k]);
    }
    const double tol = 2.220446049250313e-16 * (m > n ? m : n) * smax;
    for (int k = 0; k < n; ++k) {
        if (!(sig[k] > tol)) continue;
        double ub = 0.0;  // u_k . b, u_k = A[:, k] / sigma_k
        for (int i = 0; i < m; ++i) ub += A[(size_t)k * m + i] * b[i];
        const double w = ub / (sig[k] * sig[k]);
        for (int j = 0; j < n; ++j) x[j] += V[(size_t)k * n + j] * w;
    }
    return x;
}

}  // namespace

// Project the electric fields (and neutralise the charges through the Higgs
// momenta) of an FP64 [36][S] device state in place: `iters` iterations.
int ewpt_gauss_project_fp64(const Grid& g, const ewpt_params& p, double* y, int iters, cudaStream_t st,
                            std::string* err) {
    if (iters <= 0) return EWPT_OK;
    const int hx = g.nx / 2 + 1;
    const int64_t H = (int64_t)hx * g.ny * g.nz;
    cufftHandle fwd = 0, inv = 0;
    if (cufftPlan3d(&fwd, g.nz, g.ny, g.nx, CUFFT_D2Z) != CUFFT_SUCCESS ||
        cufftPlan3d(&inv, g.nz, g.ny, g.nx, CUFFT_Z2D) != CUFFT_SUCCESS) {
        if (fwd) cufftDestroy(fwd);
        *err = "cufftPlan3d (D2Z/Z2D) failed";
        return EWPT_ERR_CUFFT;
    }
    cufftSetStream(fwd, st);
    cufftSetStream(inv, st);
    // squared symbol per axis; |s|^2 cut: 1e-12 of its largest value (the sum
    // of each axis' largest)
    const int N[3] = {g.nx, g.ny, g.nz};
    std::vector<double> sym((size_t)g.nx + g.ny + g.nz);
    double smax = 0.0;
    for (int d = 0, o = 0; d < 3; o += N[d++]) {
        double m = 0.0;
        for (int n = 0; n < N[d]; ++n) {
            sym[o + n] = std::pow(host_symbol(6.283185307179586 * n / N[d], p.dx), 2);
            m = std::fmax(m, sym[o + n]);
        }
        smax += m;
    }
    const double cut = 1e-12 * smax, t = 1.0 / (60.0 * p.dx);
    // src [4][Sp] (the source, then chi), one half spectrum, the symbol's tables, the moments
    const size_t npart = (size_t)kMomentBlocks * 2 * kND;
    double *src = nullptr, *tab = nullptr;
    cufftDoubleComplex* C = nullptr;
    const int64_t Sp = (g.S + 1) / 2 * 2;  // array stride: cuFFT wants its arrays aligned to a complex number
    cudaError_t e = cudaMallocAsync(&src, (size_t)4 * Sp * 8, st);
    if (e == cudaSuccess) e = cudaMallocAsync(&C, (size_t)H * sizeof(cufftDoubleComplex), st);
    if (e == cudaSuccess) e = cudaMallocAsync(&tab, (sym.size() + npart + 8 * kND) * 8, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(tab, sym.data(), sym.size() * 8, cudaMemcpyHostToDevice, st);
    double* const part = tab + sym.size();
    const std::vector<int> es = null_vectors(g);
    const int ne = (int)es.size(), n = 4 * ne;
    const unsigned sites = (unsigned)((g.S + 127) / 128);
    const double coup[4] = {p.gw, p.gw, p.gw, p.gy};
    bool fft_ok = true;
    for (int it = 0; it < iters && e == cudaSuccess && fft_ok; ++it) {
        // 1. neutralise the charges' null-mode components
        double hs[8 * kND], sums[8 * kNQ] = {};
        k_class_moments<<<kMomentBlocks, 32 * kMomentWarps, 0, st>>>(g, y, p.gw, p.gy, part);
        k_fold_moments<<<1, 1024, 0, st>>>(part, part + npart);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(hs, part + npart, sizeof hs, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) break;
        for (int c = 0; c < 8; ++c) {
            double* v = sums + c * kNQ;
            const double* h = hs + c * kND;
            for (int a = 0; a < 4; ++a) {
                v[a] = h[a];
                v[4 + 4 * a + a] = coup[a] * h[4];
            }
            for (int a = 0; a < 3; ++a) {
                v[4 + 4 * a + 3] = coup[a] * h[5 + a];
                v[4 + 4 * 3 + a] = coup[3] * h[5 + a];
            }
        }
        std::vector<double> A((size_t)n * n), Q(n);
        for (int a = 0; a < 4; ++a) {
            for (int i = 0; i < ne; ++i) Q[a * ne + i] = -moment(&sums[a], kNQ, es[i]);
            for (int b = 0; b < 4; ++b)
                for (int i = 0; i < ne; ++i)
                    for (int j = 0; j < ne; ++j)
                        A[(size_t)(a * ne + i) * n + b * ne + j] = moment(&sums[4 + 4 * a + b], kNQ, es[i] ^ es[j]);
        }
        const std::vector<double> alpha = lstsq(A, n, n, Q);
        Table32 shift;
        for (int b = 0; b < 4; ++b)
            for (int c = 0; c < 8; ++c) {
                double w = 0.0;
                for (int j = 0; j < ne; ++j) w += alpha[b * ne + j] * (__builtin_popcount(c & es[j]) & 1 ? -1.0 : 1.0);
                shift.t[b * 8 + c] = w;
            }
        // 2. sources of this iteration, then each group's projection
        k_source<<<sites, 128, 0, st>>>(g, y, shift, p.gw, p.gy, t, src, Sp);
        e = cudaGetLastError();
        for (int grp = 0; grp < 4 && e == cudaSuccess && fft_ok; ++grp) {
            double* f = src + (size_t)grp * Sp;
            fft_ok = cufftExecD2Z(fwd, f, C) == CUFFT_SUCCESS;
            if (!fft_ok) break;
            k_solve<<<1216, 256, 0, st>>>(g, tab, tab + g.nx, tab + g.nx + g.ny, cut, C);
            e = cudaGetLastError();
            if (e == cudaSuccess) fft_ok = cufftExecZ2D(inv, C, f) == CUFFT_SUCCESS;
        }
        if (e == cudaSuccess && fft_ok) {
            k_subtract<<<sites, 128, 0, st>>>(g, y, src, Sp, t);
            e = cudaGetLastError();
        }
    }
    const cudaError_t ef[3] = {src ? cudaFreeAsync(src, st) : cudaSuccess, C ? cudaFreeAsync(C, st) : cudaSuccess,
                               tab ? cudaFreeAsync(tab, st) : cudaSuccess};
    for (cudaError_t x : ef)
        if (e == cudaSuccess) e = x;
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cufftDestroy(fwd);
    cufftDestroy(inv);
    if (!fft_ok) {
        *err = "cuFFT execution failed";
        return EWPT_ERR_CUFFT;
    }
    if (e != cudaSuccess) {
        *err = cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? EWPT_ERR_OOM : EWPT_ERR_CUDA;
    }
    return EWPT_OK;
}

extern "C" int ewpt_gauss_project(ewpt_ctx* c, int32_t iters) {
    if (!c) return ewpt_fail(nullptr, EWPT_ERR_ARG, "ctx is NULL");
    if (iters < 0) return ewpt_fail(c, EWPT_ERR_ARG, "iterations < 0");
    if (c->view || c->slab) return ewpt_fail(c, EWPT_ERR_STATE, "needs a whole-lattice context");
    if (c->p.stencil_order != 6) return ewpt_fail(c, EWPT_ERR_ARG, "the projection uses the 6th-order stencil");
    cudaSetDevice(c->p.device);
    // the FP64 state, or the FP32/DF64 form's state joined into FP64
    const double* cur;
    int rc = ewpt_state64(c, &cur);
    if (rc) return rc;
    double* y = const_cast<double*>(cur);
    std::string err;
    rc = ewpt_gauss_project_fp64(c->g, c->p, y, iters, c->st, &err);
    if (rc) return ewpt_fail(c, rc, "gauss_project: %s", err.c_str());
    cudaError_t e = cudaSuccess;
    if (c->p.precision == EWPT_DF64) {
        // the pairs were joined into scratch64; they are made again in place in c->y
        e = cudaMemcpyAsync(c->y, y, (size_t)36 * c->g.S * 8, cudaMemcpyDeviceToDevice, c->st);
        if (e == cudaSuccess) e = ewpt_commit_staged(c, c->y);
    } else if (c->p.precision == EWPT_FP32) {
        e = ewpt_commit_staged(c, y);  // split into hi/lo with the ghost images
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->st);
    return ewpt_cuda_check(c, e, "gauss_project");
}
