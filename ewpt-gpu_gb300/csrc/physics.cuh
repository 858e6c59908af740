// physics.cuh -- per-site right-hand side of the temporal-gauge SU(2)xU(1)
// Higgs system, templated on the arithmetic type T: double (the FP64 form's
// alternative stencil orders; its 6th-order stages spread the same equations
// over four warps, stage_fp64.cu), double-float and pairs of it (DF64).  The
// FP32 forms keep an order of operations of their own (physics_fp32.cuh).
//
// Same equations as rk4_step! (gpu-kernels-rk4/main_rk4.jl:52-661):
//   covariant derivatives  cov_derivs_temporal.jl:23-130
//   field strengths        field_strengths.jl:34-311
//   kt_phi_a               main_rk4.jl:337-407
//   kt_W_a_i               main_rk4.jl:409-560
//   kt_Y_i                 main_rk4.jl:562-581
//   k_field = momentum     main_rk4.jl:585-600
//   k_Gamma_a, k_Sigma     main_rk4.jl:603-655
// evaluated in a register-frugal order: every rate is affine in the spatial
// derivatives, so each array's gradient and Laplacian are taken together and
// folded into the rate accumulators right away (Higgs block, then one colour
// of W at a time, then Y), and each rate is handed to the sink as soon as it
// is final.  The reference's index pattern of the beta_W bracket of kt_phi
// (dW_1_3_dt, dW_1_4_dt in all three colour rows, main_rk4.jl:350-352) and
// the per-component damping term gamma*phi_a*(phi_a*pi_a)/|Phi|^2 (:349, with
// its 0/0 at |Phi| = 0) are kept.
//
// For (a, b, c) a cyclic permutation of the colours, the SU(2) rate reads
//   kt W^a_i = lap W^a_i - g sum_j (d_j W^b_i W^c_j - d_j W^c_i W^b_j)
//              - g sum_j (W^b_j F^c_ij - W^c_j F^b_ij) + J^a_i - d_i Gamma^a
//              - g (W^b_i Gamma^c - W^c_i Gamma^b) + beta terms
// which is kt_W_1_2 .. kt_W_3_4 of main_rk4.jl:409-560 term by term.
//
// Accessor `Acc`:  v(a)  value of array a (0..35, order of ewpt.h) at the site
//   grad(a, gx, gy, gz)            6th-order first derivatives
//   grad_lap(a, gx, gy, gz, lap)   first derivatives and Laplacian
//   div3(a)                        dx(a) + dy(a+1) + dz(a+2)
// Sink `out(a, rate)` receives rate a = d y_a / dt exactly once.
//
// PART splits the work between three launches when there are no beta terms:
// 0 = everything; 1 = the Higgs rates (20-23), handing the Higgs currents of
// kt W and kt Y to the sink (out.keep_current(3 a + i, J^a_i), slots 0-8;
// out.keep_current(9 + i, J^Y_i), slots 9-11); 2 = the SU(2) rates (24-32);
// 3 = the field, auxiliary and U(1) rates (0-19, 33-35).  Parts 2 and 3
// take the currents back (out.load_current).  The values are those of
// PART 0.
#pragma once

// Qualifier of the per-site arithmetic (here and in accessors.cuh).  The
// library compiles it for the device only; the test suite (oracle/devphys.cu,
// oracle/devstage.cc) defines it as inline to run the same templates on the
// host, with an operator-counting scalar type among others.
#ifndef EWPT_ARITH
#define EWPT_ARITH __device__ __forceinline__
#endif

// hgy, gp2, lam2, hJex and gam are read by no kernel now; without them the others
// lie elsewhere in the kernels' arguments and the FP32 steps take 0.3% longer
// (160^3 compensated 35.07 -> 35.19 ms per ten steps, 48^3 2.306 -> 2.314 per twenty).
template <typename T>
struct PhysCoef {
    T gw, gy, hgw, hgy;  // g, g', g/2, g'/2
    T gp2, omgp2;        // gp2, 1-gp2
    T lam2, vev2;        // 2*lambda, vev^2
    T bW, bY, bW2, bY2;  // beta_W, beta_Y, 2*beta_W, 2*beta_Y
    T hJex, gam;         // Jex/2, damping gamma
    // derived, for rates accumulated in units of the couplings
    T gg, ggy;           // gp2*g, gp2*g'
    T lam2h, hJexh, gamh;// 2*lambda, Jex/2 and gamma over g/2
    T ryw, igw;          // g'/g, 1/g
};

// Covariant derivatives D_i phi_a (cov_derivs_temporal.jl:23-130) along one
// axis with gauge components W1 = W_1_i, W2 = W_2_i and the sums Zp = W_3_i +
// Yr, Zm = W_3_i - Yr with the hypercharge component in units of g, Yr =
// (g'/g) Y_i, so that D = d + (g/2) (W terms + Yr terms).
template <typename T>
EWPT_ARITH void cov_deriv_s(T d1, T d2, T d3, T d4, T p1, T p2, T p3, T p4, T W1, T W2, T Zp, T Zm, T hgw, T& D1,
                            T& D2, T& D3, T& D4) {
    D1 = d1 + hgw * (W1 * p4 - W2 * p3 + Zp * p2);
    D2 = d2 - hgw * (W1 * p3 + W2 * p4 + Zp * p1);
    D3 = d3 + hgw * (W1 * p2 + W2 * p1 - Zm * p4);
    D4 = d4 - hgw * (W1 * p1 - W2 * p2 - Zm * p3);
}

template <typename T, bool BETA, class Acc, class Sink, int PART = 0>
EWPT_ARITH void site_rates(const Acc& A, const PhysCoef<T>& c, Sink& out) {
    static_assert(PART == 0 || !BETA, "the beta terms couple every block: PART 0 only");
    constexpr bool kHiggs = PART == 0 || PART == 1, kSU2 = PART == 0 || PART == 2,
                   kRest = PART == 0 || PART == 3;
    const T hgw = c.hgw;
    const T p1 = A.v(0), p2 = A.v(1), p3 = A.v(2), p4 = A.v(3);
    T W[3][3];  // W[a][i] = W_{a+1}_{i+2}
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int i = 0; i < 3; ++i) W[a][i] = A.v(4 + 3 * a + i);
    const T Y2 = A.v(13), Y3 = A.v(14), Y4 = A.v(15);
    const T G[3] = {A.v(16), A.v(17), A.v(18)}, S = A.v(19);
    const T pt1 = A.v(20), pt2 = A.v(21), pt3 = A.v(22), pt4 = A.v(23);

    // ---- k_field = momentum (main_rk4.jl:585-600)
    if constexpr (kRest) {
#pragma unroll
        for (int a = 0; a < 16; ++a) out(a, A.v(20 + a));
    }

    // ---- k_Gamma_a, k_Sigma (main_rk4.jl:603-655): (1 - gp2) d_i pi^a_i + gp2 g rho^a
    if constexpr (kRest) {
        T Wt[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) Wt[a][i] = A.v(24 + 3 * a + i);
        const T q12 = p1 * pt2 - p2 * pt1, q34 = p3 * pt4 - p4 * pt3;  // of charge 3 and the hypercharge
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = (a + 1) % 3, cc = (a + 2) % 3;
            // Higgs charge, then the gauge charge -(W^b . Wt^c - W^c . Wt^b)
            T q;
            if (a == 0) q = p1 * pt4 - p4 * pt1 + p3 * pt2 - p2 * pt3;
            else if (a == 1) q = p3 * pt1 - p1 * pt3 + p4 * pt2 - p2 * pt4;
            else q = q12 - q34;
            q = q - W[b][0] * Wt[cc][0] + W[cc][0] * Wt[b][0] - W[b][1] * Wt[cc][1] + W[cc][1] * Wt[b][1] -
                W[b][2] * Wt[cc][2] + W[cc][2] * Wt[b][2];
            out(16 + a, c.omgp2 * A.div3(24 + 3 * a) + c.gg * q);
        }
        out(19, c.omgp2 * A.div3(33) + c.ggy * (q12 + q34));
    }

    // ---- Higgs block: gradients, covariant derivatives, kt_phi (main_rk4.jl:337-407)
    // Every rate below is one accumulator that each product term enters with
    // a single fused multiply-add: the gauge terms of kt_phi are summed in
    // units of g/2 and those of kt_W in units of g, the coupling applied once
    // at the end.  The Higgs currents jW, jY are kept in units of g and g'.
    T ktp1, ktp2, ktp3, ktp4;
    T jW[3][3], jY[3];
    T cx = T(0), cy = T(0), cz = T(0), pdot = T(0);
    if constexpr (!kHiggs) {
        if constexpr (kSU2) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int i = 0; i < 3; ++i) jW[a][i] = out.load_current(3 * a + i);
        }
        if constexpr (kRest) {
#pragma unroll
            for (int i = 0; i < 3; ++i) jY[i] = out.load_current(9 + i);
        }
    } else {
        T d1[3], d2[3], d3[3], d4[3], l1, l2, l3, l4;
        A.grad_lap(0, d1[0], d1[1], d1[2], l1);
        A.grad_lap(1, d2[0], d2[1], d2[2], l2);
        A.grad_lap(2, d3[0], d3[1], d3[2], l3);
        A.grad_lap(3, d4[0], d4[1], d4[2], l4);
        const T Yr[3] = {c.ryw * Y2, c.ryw * Y3, c.ryw * Y4};  // (g'/g) Y_i
        // W^3 and Y act alike on (phi_1, phi_2) and oppositely on (phi_3, phi_4)
        T Zp[3], Zm[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            Zp[i] = W[2][i] + Yr[i];
            Zm[i] = W[2][i] - Yr[i];
        }
        T D1[3], D2[3], D3[3], D4[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            cov_deriv_s(d1[i], d2[i], d3[i], d4[i], p1, p2, p3, p4, W[0][i], W[1][i], Zp[i], Zm[i], hgw, D1[i],
                        D2[i], D3[i], D4[i]);
        // Higgs currents of kt_W (main_rk4.jl:415,432,449,...) and kt_Y (:563), over g and g'
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            jW[0][i] = p1 * D4[i] - p2 * D3[i] + p3 * D2[i] - p4 * D1[i];
            jW[1][i] = -p1 * D3[i] - p2 * D4[i] + p3 * D1[i] + p4 * D2[i];
            const T j12 = p1 * D2[i] - p2 * D1[i], j34 = p3 * D4[i] - p4 * D3[i];
            jW[2][i] = j12 - j34;
            jY[i] = j12 + j34;
        }
        if constexpr (PART == 1) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int i = 0; i < 3; ++i) out.keep_current(3 * a + i, jW[a][i]);
#pragma unroll
            for (int i = 0; i < 3; ++i) out.keep_current(9 + i, jY[i]);
        }
        if (BETA) {
            pdot = pt1 * p1 + pt2 * p2 + pt3 * p3 + pt4 * p4;
            cx = d1[0] * p1 + d2[0] * p2 + d3[0] * p3 + d4[0] * p4;
            cy = d1[1] * p1 + d2[1] * p2 + d3[1] * p3 + d4[1] * p4;
            cz = d1[2] * p1 + d2[2] * p2 + d3[2] * p3 + d4[2] * p4;
        }
        // The gauge terms of kt_phi pair each gradient with its covariant
        // derivative, (g/2) W.d phi + (g/2) W.D phi (main_rk4.jl:337-407), so
        // they are taken once on the sums e = d + D (d is not needed after).
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            d1[i] += D1[i];
            d2[i] += D2[i];
            d3[i] += D3[i];
            d4[i] += D4[i];
        }
        const T mag = p1 * p1 + p2 * p2 + p3 * p3 + p4 * p4;
        // over g/2: the potential and external source 2 lambda (|Phi|^2 - v^2) + Jex/2,
        // the damping gamma / |Phi|^2 (its 0/0 at |Phi| = 0 kept), the charges (g Gamma^3 +- g' Sigma)/2
        const T potg = c.lam2h * (mag - c.vev2) + c.hJexh;
        const T damp = c.gamh / mag;
        const T q12 = G[2] + c.ryw * S, q34 = c.ryw * S - G[2];
        T a1 = W[0][0] * d4[0] + W[0][1] * d4[1] + W[0][2] * d4[2] - W[1][0] * d3[0] - W[1][1] * d3[1] -
               W[1][2] * d3[2] + Zp[0] * d2[0] + Zp[1] * d2[1] + Zp[2] * d2[2] + q12 * p2 - G[1] * p3 + G[0] * p4 -
               potg * p1 - damp * p1 * (p1 * pt1);
        T a2 = -W[0][0] * d3[0] - W[0][1] * d3[1] - W[0][2] * d3[2] - W[1][0] * d4[0] - W[1][1] * d4[1] -
               W[1][2] * d4[2] - Zp[0] * d1[0] - Zp[1] * d1[1] - Zp[2] * d1[2] - q12 * p1 - G[0] * p3 - G[1] * p4 -
               potg * p2 - damp * p2 * (p2 * pt2);
        T a3 = W[0][0] * d2[0] + W[0][1] * d2[1] + W[0][2] * d2[2] + W[1][0] * d1[0] + W[1][1] * d1[1] +
               W[1][2] * d1[2] - Zm[0] * d4[0] - Zm[1] * d4[1] - Zm[2] * d4[2] + q34 * p4 + G[1] * p1 + G[0] * p2 -
               potg * p3 - damp * p3 * (p3 * pt3);
        T a4 = -W[0][0] * d1[0] - W[0][1] * d1[1] - W[0][2] * d1[2] + W[1][0] * d2[0] + W[1][1] * d2[1] +
               W[1][2] * d2[2] + Zm[0] * d3[0] + Zm[1] * d3[1] + Zm[2] * d3[2] - q34 * p3 - G[0] * p1 + G[1] * p2 -
               potg * p4 - damp * p4 * (p4 * pt4);
        ktp1 = l1 + hgw * a1;
        ktp2 = l2 + hgw * a2;
        ktp3 = l3 + hgw * a3;
        ktp4 = l4 + hgw * a4;
    }

    // ---- SU(2) block, one colour at a time (field_strengths.jl:34-224)
    //   kt W^a_i = lap W^a_i - d_i Gamma^a + g Q^a_i, Q accumulated over g.
    // The terms of colour b's derivatives and field strength in the other two
    // colours share their factors W_j, so they enter as E_ij = F^b_ij - d_j W^b_i:
    //   Q^{b-1}_i += sum_j W^{b+1}_j E_ij,   Q^{b+1}_i -= sum_j W^{b-1}_j E_ij
    T ktW[3][3];
    T F[3][3];  // beta terms only: F[b][0] = F^b_xy (W_b_23), [1] = F^b_xz (W_b_24), [2] = F^b_yz (W_b_34)
    if constexpr (kSU2) {
        T Q[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = (a + 1) % 3, cc = (a + 2) % 3;
#pragma unroll
            for (int i = 0; i < 3; ++i) Q[a][i] = jW[a][i] - W[b][i] * G[cc] + W[cc][i] * G[b];
        }
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            T dW[3][3];  // dW[i][j] = d_j W^b_i
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                T lap;
                A.grad_lap(4 + 3 * b + i, dW[i][0], dW[i][1], dW[i][2], lap);
                Q[b][i] = Q[b][i] + lap * c.igw;
            }
            const int b1 = (b + 1) % 3, b2 = (b + 2) % 3;
#pragma unroll
            for (int i = 0; i < 3; ++i) {  // E_ii = -d_i W^b_i
                Q[b2][i] = Q[b2][i] - W[b1][i] * dW[i][i];
                Q[b1][i] = Q[b1][i] + W[b2][i] * dW[i][i];
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const int i = m == 2 ? 1 : 0, j = m == 0 ? 1 : 2;
                const T Fij = dW[j][i] - dW[i][j] + c.gw * (W[b1][i] * W[b2][j] - W[b1][j] * W[b2][i]);
                if (BETA) F[b][m] = Fij;
                const T Eij = Fij - dW[i][j], mEji = Fij + dW[j][i];  // E_ij and -E_ji
                Q[b2][i] = Q[b2][i] + W[b1][j] * Eij;
                Q[b1][i] = Q[b1][i] - W[b2][j] * Eij;
                Q[b2][j] = Q[b2][j] - W[b1][i] * mEji;
                Q[b1][j] = Q[b1][j] + W[b2][i] * mEji;
            }
        }
        // the coupling and the auxiliary gradient
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            T g[3];
            A.grad(16 + a, g[0], g[1], g[2]);
#pragma unroll
            for (int i = 0; i < 3; ++i) ktW[a][i] = c.gw * Q[a][i] - g[i];
        }
    }

    // ---- U(1) block (field_strengths.jl:281-311, main_rk4.jl:562-581)
    T ktY[3], FY[3];
    if constexpr (kRest) {
        T dY[3][3], lap[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) A.grad_lap(13 + i, dY[i][0], dY[i][1], dY[i][2], lap[i]);
        FY[0] = dY[1][0] - dY[0][1];
        FY[1] = dY[2][0] - dY[0][2];
        FY[2] = dY[2][1] - dY[1][2];
        T g[3];
        A.grad(19, g[0], g[1], g[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) ktY[i] = lap[i] + c.gy * jY[i] - g[i];
    }

    // ---- beta (CP-odd) terms
    if (BETA) {
        T Wt[3][3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) Wt[a][i] = A.v(24 + 3 * a + i);
        const T Yt2 = A.v(33), Yt3 = A.v(34), Yt4 = A.v(35);
        // dual field strength: B_x = F_yz, B_y = -F_xz, B_z = F_xy
        const T bWt = (Wt[0][0] * F[0][2] + Wt[0][1] * (-F[0][1]) + Wt[0][2] * F[0][0] +
                       Wt[1][0] * F[1][2] + Wt[0][1] * (-F[1][1]) + Wt[0][2] * F[1][0] +
                       Wt[2][0] * F[2][2] + Wt[0][1] * (-F[2][1]) + Wt[0][2] * F[2][0]);
        const T bYt = (Yt2 * FY[2] + Yt3 * (-FY[1]) + Yt4 * FY[0]);
        const T bsum = c.bW * bWt + c.bY * bYt;
        ktp1 += bsum * p1;
        ktp2 += bsum * p2;
        ktp3 += bsum * p3;
        ktp4 += bsum * p4;
        const T bwp = c.bW2 * pdot, byp = c.bY2 * pdot;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            ktW[a][0] += -bwp * F[a][2] + c.bW2 * (cy * Wt[a][2] - cz * Wt[a][1]);
            ktW[a][1] += bwp * F[a][1] + c.bW2 * (cz * Wt[a][0] - cx * Wt[a][2]);
            ktW[a][2] += -bwp * F[a][0] + c.bW2 * (cx * Wt[a][1] - cy * Wt[a][0]);
        }
        ktY[0] += -byp * FY[2] + c.bY2 * (cy * Yt4 - cz * Yt3);
        ktY[1] += byp * FY[1] + c.bY2 * (cz * Yt2 - cx * Yt4);
        ktY[2] += -byp * FY[0] + c.bY2 * (cx * Yt3 - cy * Yt2);
    }
    if constexpr (kHiggs) {
        out(20, ktp1);
        out(21, ktp2);
        out(22, ktp3);
        out(23, ktp4);
    }
    if constexpr (kSU2) {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) out(24 + 3 * a + i, ktW[a][i]);
    }
    if constexpr (kRest) {
        out(33, ktY[0]);
        out(34, ktY[1]);
        out(35, ktY[2]);
    }
}

// PART 1 axis by axis, for arithmetic types whose values take several
// registers: the gradients of one axis at a time, each Laplacian at the end.
// The same terms as in site_rates, summed in another order.  Accessor:
// d1(a, i) and lap(a).
template <typename T, class Acc, class Sink>
EWPT_ARITH void higgs_rates_by_axis(const Acc& A, const PhysCoef<T>& c, Sink& out) {
    const T p[4] = {A.v(0), A.v(1), A.v(2), A.v(3)};
    T a[4];  // kt_phi over g/2, without the Laplacian
    {
        const T mag = p[0] * p[0] + p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
        const T potg = c.lam2h * (mag - c.vev2) + c.hJexh;
        const T damp = c.gamh / mag;
        const T G1 = A.v(16), G2 = A.v(17), G3 = A.v(18), S = c.ryw * A.v(19);
        const T q12 = G3 + S, q34 = S - G3;
        a[0] = q12 * p[1] - G2 * p[2] + G1 * p[3] - potg * p[0] - damp * p[0] * (p[0] * A.v(20));
        a[1] = -q12 * p[0] - G1 * p[2] - G2 * p[3] - potg * p[1] - damp * p[1] * (p[1] * A.v(21));
        a[2] = q34 * p[3] + G2 * p[0] + G1 * p[1] - potg * p[2] - damp * p[2] * (p[2] * A.v(22));
        a[3] = -q34 * p[2] - G1 * p[0] + G2 * p[1] - potg * p[3] - damp * p[3] * (p[3] * A.v(23));
    }
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
        const T W1 = A.v(4 + i), W2 = A.v(7 + i), W3 = A.v(10 + i), Yr = c.ryw * A.v(13 + i);
        const T Zp = W3 + Yr, Zm = W3 - Yr;
        T d1 = A.d1(0, i), d2 = A.d1(1, i), d3 = A.d1(2, i), d4 = A.d1(3, i), D1, D2, D3, D4;
        cov_deriv_s(d1, d2, d3, d4, p[0], p[1], p[2], p[3], W1, W2, Zp, Zm, c.hgw, D1, D2, D3, D4);
        out.keep_current(i, p[0] * D4 - p[1] * D3 + p[2] * D2 - p[3] * D1);
        out.keep_current(3 + i, -p[0] * D3 - p[1] * D4 + p[2] * D1 + p[3] * D2);
        const T j12 = p[0] * D2 - p[1] * D1, j34 = p[2] * D4 - p[3] * D3;
        out.keep_current(6 + i, j12 - j34);
        out.keep_current(9 + i, j12 + j34);
        d1 += D1;
        d2 += D2;
        d3 += D3;
        d4 += D4;
        a[0] += W1 * d4 - W2 * d3 + Zp * d2;
        a[1] -= W1 * d3 + W2 * d4 + Zp * d1;
        a[2] += W1 * d2 + W2 * d1 - Zm * d4;
        a[3] -= W1 * d1 - W2 * d2 - Zm * d3;
    }
#pragma unroll 1
    for (int b = 0; b < 4; ++b) out(20 + b, A.lap(b) + c.hgw * (b == 0 ? a[0] : b == 1 ? a[1] : b == 2 ? a[2] : a[3]));
}
