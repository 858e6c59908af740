// devstage.cc -- the library's per-site code for the host, by a host C++
// compiler (test infrastructure, never linked into libewpt):
//  * the 6th-order FP64 stages (csrc/stage_fp64.cuh), the four warps of a site
//    as threads;
//  * their integer stencils and those of the diagnostics (csrc/fixstencil.cuh);
//  * the equations of the FP32 forms (csrc/physics_fp32.cuh) in FP64, and those
//    of the DF64 form and of the alternative stencil orders (csrc/physics.cuh).
#include <condition_variable>
#include <mutex>
#include <thread>

#include "host_device.h"  // after the standard headers, which use its attribute's name

#include "fixstencil.cuh"
#include "physics_fp32.cuh"
#include "stage_fp64.cuh"

namespace {

// bar.arrive and bar.sync of `n` threads
struct Barrier {
    int n, waiting = 0;
    long phase = 0;
    std::mutex m{};
    std::condition_variable cv{};
    void arrive(bool wait) {
        std::unique_lock<std::mutex> l(m);
        const long p = phase;
        if (++waiting == n) {
            waiting = 0;
            ++phase;
            cv.notify_all();
        } else if (wait) {
            cv.wait(l, [&] { return phase != p; });
        }
    }
};
Barrier g_parts{kWarps}, g_colours{kWarps - 1}, g_site{kWarps};

void parts_written() { g_parts.arrive(false); }
void parts_ready() { g_parts.arrive(true); }
void colours_ready() { g_colours.arrive(true); }

template <class F>
void sites(int nx, int ny, int nz, F f) {
    for (int k = 0; k < nz; ++k)
        for (int j = 0; j < ny; ++j)
            for (int i = 0; i < nx; ++i) f(i, j, k, i + nx * (j + ny * k));
}

Grid box(int nx, int ny, int nz) { return Grid{nx, ny, nz, (int64_t)nx * ny * nz}; }

ewpt_params params(const double* cp) {
    ewpt_params p{};
    p.gw = cp[0];
    p.gy = cp[1];
    p.gp2 = cp[2];
    p.lambda = cp[3];
    p.vev = cp[4];
    p.beta_w = cp[5];
    p.beta_y = cp[6];
    p.dx = cp[7];
    return p;
}

template <bool BETA>
void rates_fp64(const Grid& g, const Ptr36& X, const Coef& pc, const RatesOut& out) {
    SharedOf<BETA> sh;
    auto role = [&](int warp) {
        sites(g.nx, g.ny, g.nz, [&](int i, int j, int k, int c) {
            FixAcc A{X, g};
            A.place(i, j, k);
            const int lane = c % kSites;
            stencils(A, sh, lane, warp);
            g_site.arrive(true);
            if (warp == 0)
                higgs_warp<0, BETA>(A, pc, sh, lane, true, out);
            else
                colour_warp<0, BETA>(A, pc, sh, lane, true, warp - 1, out);
            g_site.arrive(true);
        });
    };
    std::thread t[kWarps];
    for (int w = 0; w < kWarps; ++w) t[w] = std::thread(role, w);
    for (std::thread& w : t) w.join();
}

struct RateSink {
    double* r;
    int64_t S, c;
    void operator()(int a, double v) { r[a * S + c] = v; }
};

}  // namespace

extern "C" {

// All 36 rates at every site, y and r [36][S]; cp: gw, gy, gp2, lambda, vev,
// beta_w, beta_y, dx.  form 0: the FP64 stages; 1: physics_fp32.cuh, 2:
// physics.cuh over the FP64 accessor.
void ds_rates(int nx, int ny, int nz, const double* cp, const double* y, double* r, double Jex, double gam, int form) {
    const Grid g = box(nx, ny, nz);
    const ewpt_params p = params(cp);
    const bool beta = p.beta_w != 0.0 || p.beta_y != 0.0;
    const Ptr36 X = arrays36(y, g.S);
    if (form == 0) {
        const Coef pc = make_coef(p, Jex, gam);
        const RatesOut out{arrays36(r, g.S), {1.0, pc.hgw_o, pc.gw_o}};
        beta ? rates_fp64<true>(g, X, pc, out) : rates_fp64<false>(g, X, pc, out);
        return;
    }
    const PhysCoef<double> pc = make_phys<double>(p, Jex, gam);
    sites(nx, ny, nz, [&](int i, int j, int k, int c) {
        SiteAcc<double, double, SrcPtr36<double>> A{{X}};
        A.place(i, j, k, nx, ny, nz);
        A.s = make_stencil<double>(p.dx);
        RateSink out{r, g.S, c};
        if (form == 1)
            beta ? site_rates_fp32<double, true>(A, pc, out) : site_rates_fp32<double, false>(A, pc, out);
        else
            beta ? site_rates<double, true>(A, pc, out) : site_rates<double, false>(A, pc, out);
    });
}

// The stage kernels' stencils of arrays a, a + 1, a + 2 of y [36][S]:
// out[0..3] = 60 dx grad and 180 dx^2 lap of array a by grad_lap, [4..6] = 60 dx
// grad by grad, [7] = 60 dx (d_x a + d_y (a + 1) + d_z (a + 2)).
void ds_stencils(int nx, int ny, int nz, const double* y, int a, double* out) {
    const Grid g = box(nx, ny, nz);
    Ptr36 X;
    for (int q = 0; q < 36; ++q) X.p[q] = y + q * g.S;
    sites(nx, ny, nz, [&](int i, int j, int k, int c) {
        FixAcc A{X, g};
        A.place(i, j, k);
        double* o = out + c;
        A.grad_lap(a, o[0], o[g.S], o[2 * g.S], o[3 * g.S]);
        A.grad(a, o[4 * g.S], o[5 * g.S], o[6 * g.S]);
        o[7 * g.S] = A.div3(a);
    });
}

// The diagnostics': out[0..2] = grad a, [3] = the divergence, [4..6] = the curls
// d_y (a + 2) - d_z (a + 1), d_z a - d_x (a + 2), d_x (a + 1) - d_y a.
void ds_diffs(int nx, int ny, int nz, const double* y, int a, double* out) {
    const Grid g = box(nx, ny, nz);
    sites(nx, ny, nz, [&](int i, int j, int k, int c) {
        FixDiff A;
        A.y = y;
        A.S = g.S;
        A.c = c;
        axis_offsets(i, nx, 1, A.o[0]);
        axis_offsets(j, ny, nx, A.o[1]);
        axis_offsets(k, nz, nx * ny, A.o[2]);
        double* o = out + c;
        A.grad(a, o[0], o[g.S], o[2 * g.S]);
        o[3 * g.S] = A.div(a);
        o[4 * g.S] = A.curl(a + 2, 1, a + 1, 2);
        o[5 * g.S] = A.curl(a, 2, a + 2, 0);
        o[6 * g.S] = A.curl(a + 1, 0, a, 1);
    });
}

}  // extern "C"
