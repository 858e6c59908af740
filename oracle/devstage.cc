// devstage.cc -- the library's per-site code for the host, by a host C++
// compiler (test infrastructure, never linked into libewpt): the integer FP64
// stencils of the stage kernels and of the diagnostics (csrc/fixstencil.cuh).
#include "host_device.h"

#include "fixstencil.cuh"

namespace {

template <class F>
void sites(int nx, int ny, int nz, F f) {
    for (int k = 0; k < nz; ++k)
        for (int j = 0; j < ny; ++j)
            for (int i = 0; i < nx; ++i) f(i, j, k, i + nx * (j + ny * k));
}

Grid box(int nx, int ny, int nz) { return Grid{nx, ny, nz, (int64_t)nx * ny * nz}; }

}  // namespace

extern "C" {

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
