// channel_kernels.cuh - column kernels of one RK3 substep of the LittleHarsh channel DNS (sm_100a):
// right-hand sides, thread-per-column solves, mean mode, layout conversion, strided transforms.
// Device layout and transform passes: transform_kernels.cuh.
#pragma once

#include "transform_kernels.cuh"

namespace cfd {

// --------------------------------------------------------------------------------------
// Column kernel: RHS0_u1/u2/u3 (littleharsh.f90:613-730), the tail of nonlinear
// (der_x/der_z FOU3D.f90:310-414 as ik products with the kz = -N2/2 row zeroed,
// der_yu_h/der_yv_h :453-493, du += -g Nu :233-244) and the solveU/solveV prologue
// (du = u + dt du, wall/ghost rows 0; littleharsh.f90:744-786).
// MODE bits: 1 = RHS0, 2 = nonlinear tail, 4 = solve prologue.
// --------------------------------------------------------------------------------------
struct RKCoef {
    double C1;    // a/Re
    double C2;    // -c
    double dRK;   // d = g + c
    double mg;    // -g
    double dt;
    int krk;
    // 1: the x/z advective derivatives of every interior plane are those of the last plane
    // of the grid (top ghost centre for u/w, top wall face for v), as the reference computes
    // them with one plane slab (2-D scratch summed after the plane loop, FOU3D.f90:1541,
    // 1571-1585, 1602-1613); 0: per plane
    int lastplane;
};

template <typename T2> __device__ __forceinline__ T2 ldT(const T2* p) { return *p; }

template <typename T2, int MODE>
__global__ void __launch_bounds__(256, sizeof(T2) == 8 ? 3 : 0) k_rhs(Dims d, Geo g, RKCoef c, const double* __restrict__ scal,
                                             const double2* __restrict__ u1, const double2* __restrict__ u2,
                                             const double2* __restrict__ u3, const double2* __restrict__ p,
                                             T2* __restrict__ Nu1, T2* __restrict__ Nu2, T2* __restrict__ Nu3,
                                             double2* __restrict__ du1, double2* __restrict__ du2,
                                             double2* __restrict__ du3, const T2* __restrict__ S0,
                                             const T2* __restrict__ S1, const T2* __restrict__ S2,
                                             const T2* __restrict__ S3, int JC) {
    // one thread = one column and a chunk of JC planes (blockIdx.y); no recurrence in y
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int i = col % d.nkx, q = col / d.nkx;
    const double kxv = g.kx[i], kzv = g.kz[q];
    const double k2 = (-kxv * kxv) + (-kzv * kzv);
    const bool zrow = (q == d.n2 / 2);  // der_x/der_z zero the kz = -N2/2 mode
    const size_t nc = d.ncol;
    const double mpgx = scal[0];
    constexpr bool RHS0 = (MODE & 1) != 0, NL = (MODE & 2) != 0, PRO = (MODE & 4) != 0;
    const int cb = blockIdx.y;

    // ---- u and w (ugrid), j = ju0+1 .. ju1-1
    {
        const int jb = d.ju0 + 1 + cb * JC;
        const int je = min(jb + JC, d.ju1);
        if (jb < je) {
            const size_t ju = (size_t)(jb - d.ju0);
            double2 a_m = u1[(ju - 1) * nc + col], a_0 = u1[ju * nc + col];
            double2 w_m = u3[(ju - 1) * nc + col], w_0 = u3[ju * nc + col];
            const size_t vs = (size_t)d.nyu * nc;  // first v-slot
            double2 uv_m = NL ? to_d2(S0[vs + (size_t)(jb - 1 - d.jv0) * nc + col]) : dc(0, 0);
            double2 vw_m = NL ? to_d2(S1[vs + (size_t)(jb - 1 - d.jv0) * nc + col]) : dc(0, 0);
            for (int j = jb; j < je; ++j) {
                const size_t ju = (size_t)(j - d.ju0);
                const double2 a_p = u1[(ju + 1) * nc + col];
                const double2 w_p = u3[(ju + 1) * nc + col];
                const size_t jp = (size_t)(j - d.jp0);
                double2 r1, r3;
                if (RHS0) {
                    const double c0 = g.dyu2i[3 * ju + 0], c1 = g.dyu2i[3 * ju + 1], c2 = g.dyu2i[3 * ju + 2];
                    const double dg = k2 + c1;
                    const double2 Lu = dadd(dadd(dscl(c0, a_m), dscl(dg, a_0)), dscl(c2, a_p));
                    const double2 Lw = dadd(dadd(dscl(c0, w_m), dscl(dg, w_0)), dscl(c2, w_p));
                    const double2 pp = p[jp * nc + col];
                    const double2 n1o = to_d2(Nu1[ju * nc + col]);
                    const double2 n3o = to_d2(Nu3[ju * nc + col]);
                    r1 = dadd(dadd(dscl(c.C1, Lu), dscl(c.C2, n1o)), dik(-c.dRK * kxv, pp));
                    r3 = dadd(dadd(dscl(c.C1, Lw), dscl(c.C2, n3o)), dik(-c.dRK * kzv, pp));
                    if (col == 0) r1.x += -c.dRK * mpgx;
                } else {
                    r1 = du1[ju * nc + col];
                    r3 = du3[ju * nc + col];
                }
                if (NL) {
                    const size_t su = ju * nc + col;
                    const size_t sx = c.lastplane ? (size_t)(d.nyu - 1) * nc + col : su;  // x/z products
                    const size_t sv = vs + (size_t)(j - d.jv0) * nc + col;
                    const double2 uv_p = to_d2(S0[sv]), vw_p = to_d2(S1[sv]);
                    const double dth = g.dthdyu[ju];
                    double2 n1 = zrow ? dc(0, 0) : dadd(dik(kxv, to_d2(S0[sx])), dik(kzv, to_d2(S1[sx])));
                    double2 n3 = zrow ? dc(0, 0) : dadd(dik(kxv, to_d2(S1[sx])), dik(kzv, to_d2(S3[sx])));
                    n1 = dadd(n1, dscl(dth, dsub(uv_p, uv_m)));
                    n3 = dadd(n3, dscl(dth, dsub(vw_p, vw_m)));
                    Nu1[su] = to_t2<T2>(n1);
                    Nu3[su] = to_t2<T2>(n3);
                    r1 = dadd(r1, dscl(c.mg, n1));
                    r3 = dadd(r3, dscl(c.mg, n3));
                    uv_m = uv_p;
                    vw_m = vw_p;
                }
                if (PRO) {
                    r1 = dadd(a_0, dscl(c.dt, r1));
                    r3 = dadd(w_0, dscl(c.dt, r3));
                }
                du1[ju * nc + col] = r1;
                du3[ju * nc + col] = r3;
                a_m = a_0; a_0 = a_p;
                w_m = w_0; w_0 = w_p;
            }
        }
    }
    // ---- v (vgrid), j = jv0+1 .. jv1-1
    {
        const int jb = d.jv0 + 1 + cb * JC;
        const int je = min(jb + JC, d.jv1);
        if (jb < je) {
            const size_t jv = (size_t)(jb - d.jv0);
            double2 v_m = u2[(jv - 1) * nc + col], v_0 = u2[jv * nc + col];
            double2 vv_0 = NL ? to_d2(S2[(size_t)(jb - d.ju0) * nc + col]) : dc(0, 0);
            const size_t vs = (size_t)d.nyu * nc;
            for (int j = jb; j < je; ++j) {
                const size_t jv = (size_t)(j - d.jv0);
                const double2 v_p = u2[(jv + 1) * nc + col];
                double2 r2;
                if (RHS0) {
                    const double c0 = g.dyv2i[3 * jv + 0], c1 = g.dyv2i[3 * jv + 1], c2 = g.dyv2i[3 * jv + 2];
                    const double2 Lv = dadd(dadd(dscl(c0, v_m), dscl(k2 + c1, v_0)), dscl(c2, v_p));
                    const double C3 = -c.dRK * g.dthdyv[jv];
                    const double2 pa = p[(size_t)(j + 1 - d.jp0) * nc + col];
                    const double2 pb = p[(size_t)(j - d.jp0) * nc + col];
                    const double2 n2o = to_d2(Nu2[jv * nc + col]);
                    r2 = dadd(dadd(dscl(c.C1, Lv), dscl(c.C2, n2o)), dscl(C3, dsub(pa, pb)));
                } else {
                    r2 = du2[jv * nc + col];
                }
                if (NL) {
                    const size_t sv = vs + (c.lastplane ? (size_t)(d.nyv - 1) : jv) * nc + col;
                    const double2 vv_p = to_d2(S2[(size_t)(j + 1 - d.ju0) * nc + col]);
                    double2 n2 = zrow ? dc(0, 0) : dadd(dik(kxv, to_d2(S0[sv])), dik(kzv, to_d2(S1[sv])));
                    n2 = dadd(n2, dscl(g.dthdyv[jv], dsub(vv_p, vv_0)));
                    Nu2[jv * nc + col] = to_t2<T2>(n2);
                    r2 = dadd(r2, dscl(c.mg, n2));
                    vv_0 = vv_p;
                }
                if (PRO) r2 = dadd(v_0, dscl(c.dt, r2));
                du2[jv * nc + col] = r2;
                v_m = v_0; v_0 = v_p;
            }
        }
    }
    if (PRO && cb == 0) {
        du1[col] = dc(0, 0);
        du3[col] = dc(0, 0);
        du1[(size_t)(d.nyu - 1) * nc + col] = dc(0, 0);
        du3[(size_t)(d.nyu - 1) * nc + col] = dc(0, 0);
        du2[col] = dc(0, 0);
        du2[(size_t)(d.nyv - 1) * nc + col] = dc(0, 0);
    }
}

// --------------------------------------------------------------------------------------
// Implicit Helmholtz solves: LUsolU/LUsolV with LU_buildU/V + LU_dec computed on the fly
// (tridLU_3D_IB.f90:50-160, 349-413, 521-559).  One thread per (kx,kz) column; the
// forward sweep leaves y_j in the solution array and the scaled upper diagonal in `cs`.
// u and w share the matrix and its factorisation.
// --------------------------------------------------------------------------------------
// Loads of the sweeps are batched UB planes at a time so that each thread keeps several
// independent loads in flight while the recurrence runs on registers.
#define CFD_UB 8

__global__ void __launch_bounds__(256) k_solve_uvw(Dims d, Geo g, double beta, double2* __restrict__ u1,
                                                   double2* __restrict__ u2, double2* __restrict__ u3,
                                                   const double2* __restrict__ r1, const double2* __restrict__ r2,
                                                   const double2* __restrict__ r3, double* __restrict__ cs_uw,
                                                   double* __restrict__ cs_v, int part0) {
    // blockIdx.y + part0: 0 = the u/w systems, 1 = the v system
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int i = col % d.nkx, q = col / d.nkx;
    const double k2x = -g.kx[i] * g.kx[i], k2z = -g.kz[q] * g.kz[q];
    const size_t nc = d.ncol;
    if (blockIdx.y + part0 == 0) {
        // u and w share the matrix: rows (0,1,gwb), interior, (gwt,1,0)
        const int n = d.nyu;
        double dprev = 1.0, a3prev = g.gwb;
        double2 y1 = r1[col], y3 = r3[col];
        u1[col] = y1;
        u3[col] = y3;
        for (int j0 = 1; j0 < n; j0 += CFD_UB) {
            double2 ra[CFD_UB], rc[CFD_UB];
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t)
                if (j0 + t < n) { ra[t] = r1[(size_t)(j0 + t) * nc + col]; rc[t] = r3[(size_t)(j0 + t) * nc + col]; }
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t) {
                const int jj = j0 + t;
                if (jj >= n) break;
                double a1, a2, a3;
                if (jj < n - 1) {
                    a1 = -beta * g.dyu2i[3 * jj + 0];
                    a2 = 1.0 - beta * (g.dyu2i[3 * jj + 1] + k2x + k2z);
                    a3 = -beta * g.dyu2i[3 * jj + 2];
                } else {
                    a1 = g.gwt; a2 = 1.0; a3 = 0.0;
                }
                const double csm = a3prev * dprev;  // a(3,j-1) * a(2,j-1)
                cs_uw[(size_t)(jj - 1) * nc + col] = csm;
                const double dj = 1.0 / (a2 - a1 * csm);
                y1 = dscl(dj, dsub(ra[t], dscl(a1, y1)));
                y3 = dscl(dj, dsub(rc[t], dscl(a1, y3)));
                u1[(size_t)jj * nc + col] = y1;
                u3[(size_t)jj * nc + col] = y3;
                dprev = dj;
                a3prev = a3;
            }
        }
        double2 x1 = y1, x3 = y3;
        for (int j0 = n - 2; j0 >= 0; j0 -= CFD_UB) {
            double cc[CFD_UB];
            double2 ya[CFD_UB], yc[CFD_UB];
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t)
                if (j0 - t >= 0) {
                    const size_t o = (size_t)(j0 - t) * nc + col;
                    cc[t] = cs_uw[o]; ya[t] = u1[o]; yc[t] = u3[o];
                }
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t) {
                if (j0 - t < 0) break;
                const size_t o = (size_t)(j0 - t) * nc + col;
                x1 = dsub(ya[t], dscl(cc[t], x1));
                x3 = dsub(yc[t], dscl(cc[t], x3));
                u1[o] = x1;
                u3[o] = x3;
            }
        }
    } else {
        // v: identity wall rows
        const int n = d.nyv;
        double dprev = 1.0, a3prev = 0.0;
        double2 y = r2[col];
        u2[col] = y;
        for (int j0 = 1; j0 < n; j0 += CFD_UB) {
            double2 ra[CFD_UB];
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t)
                if (j0 + t < n) ra[t] = r2[(size_t)(j0 + t) * nc + col];
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t) {
                const int jj = j0 + t;
                if (jj >= n) break;
                double a1, a2, a3;
                if (jj < n - 1) {
                    a1 = -beta * g.dyv2i[3 * jj + 0];
                    a2 = 1.0 - beta * (g.dyv2i[3 * jj + 1] + k2x + k2z);
                    a3 = -beta * g.dyv2i[3 * jj + 2];
                } else {
                    a1 = 0.0; a2 = 1.0; a3 = 0.0;
                }
                const double csm = a3prev * dprev;
                cs_v[(size_t)(jj - 1) * nc + col] = csm;
                const double dj = 1.0 / (a2 - a1 * csm);
                y = dscl(dj, dsub(ra[t], dscl(a1, y)));
                u2[(size_t)jj * nc + col] = y;
                dprev = dj;
                a3prev = a3;
            }
        }
        double2 x = y;
        for (int j0 = n - 2; j0 >= 0; j0 -= CFD_UB) {
            double cc[CFD_UB];
            double2 ya[CFD_UB];
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t)
                if (j0 - t >= 0) {
                    const size_t o = (size_t)(j0 - t) * nc + col;
                    cc[t] = cs_v[o]; ya[t] = u2[o];
                }
#pragma unroll
            for (int t = 0; t < CFD_UB; ++t) {
                if (j0 - t < 0) break;
                x = dsub(ya[t], dscl(cc[t], x));
                u2[(size_t)(j0 - t) * nc + col] = x;
            }
        }
    }
}

// --------------------------------------------------------------------------------------
// solveP (littleharsh.f90:556-611): divergence (:209-244), psi = div/(dt(a+b)),
// psi(mean, bottom) = 0, LUsolP with the D.G matrix of LU_buildP/LU_decP computed on
// the fly (tridLU_3D_IB.f90:284-318, 417-491, 562-603), p += psi.
// --------------------------------------------------------------------------------------
template <bool FUSE>
__global__ void __launch_bounds__(256) k_solve_p(Dims d, Geo g, double dtirk, double2* __restrict__ u1,
                                                 double2* __restrict__ u2, double2* __restrict__ u3,
                                                 double2* __restrict__ p, double2* __restrict__ psi,
                                                 double2* __restrict__ divo, double* __restrict__ cs, double mean_diag,
                                                 double dtrk) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int i = col % d.nkx, q = col / d.nkx;
    const double kxv = g.kx[i], kzv = g.kz[q];
    const double k2x = -kxv * kxv, k2z = -kzv * kzv;
    const size_t nc = d.ncol;
    const int n = d.nyp;
    // D.G coefficients: D_b(m) = -dthdyu(m+1), G_b(m) = -dthdyv(m), D_t(m) = dthdyu(m), G_t(m) = dthdyv(m-1)
    auto DTHU = [&](int j) { return g.dthdyu[j - d.ju0]; };
    auto DTHV = [&](int j) { return g.dthdyv[j - d.jv0]; };
    double dprev = 0.0, a3prev = 0.0;
    double2 y = dc(0, 0);
    double2 vb = u2[(size_t)(d.jp0 - 1 - d.jv0) * nc + col];
    for (int jj0 = 0; jj0 < n; jj0 += CFD_UB) {
        double2 A[CFD_UB], W[CFD_UB], VA[CFD_UB];
#pragma unroll
        for (int t = 0; t < CFD_UB; ++t)
            if (jj0 + t < n) {
                const int j = d.jp0 + jj0 + t;
                A[t] = u1[(size_t)(j - d.ju0) * nc + col];
                W[t] = u3[(size_t)(j - d.ju0) * nc + col];
                VA[t] = u2[(size_t)(j - d.jv0) * nc + col];
            }
#pragma unroll
        for (int t = 0; t < CFD_UB; ++t) {
            const int jj = jj0 + t;
            if (jj >= n) break;
            const int j = d.jp0 + jj;
            // divergence at p-point j
            const double2 dv = dadd(dadd(dik(kxv, A[t]), dik(kzv, W[t])), dscl(DTHU(j), dsub(VA[t], vb)));
            vb = VA[t];
            if (divo) divo[(size_t)jj * nc + col] = dv;
            double2 r = dscl(dtirk, dv);
            double a1, a2, a3;
            if (jj == 0) {
                a1 = 0.0;
                a2 = (DTHU(j) * -DTHV(j)) + k2x + k2z;
                a3 = (DTHU(j) * DTHV(j));
                if (col == 0) { a2 = mean_diag; a3 = 0.0; r = dc(0, 0); }
            } else if (jj == n - 1) {
                a1 = (-DTHU(j)) * (-DTHV(j - 1));
                a2 = ((-DTHU(j)) * DTHV(j - 1)) + k2x + k2z;
                a3 = 0.0;
            } else {
                a2 = ((-DTHU(j)) * DTHV(j - 1)) + (DTHU(j) * -DTHV(j)) + k2x + k2z;
                a1 = ((-DTHU(j)) * (-DTHV(j - 1)));
                a3 = (DTHU(j) * DTHV(j));
            }
            double dj;
            if (jj == 0) {
                dj = 1.0 / a2;
                y = dscl(dj, r);
            } else {
                const double csm = a3prev * dprev;
                cs[(size_t)(jj - 1) * nc + col] = csm;
                dj = 1.0 / (a2 - a1 * csm);
                y = dscl(dj, dsub(r, dscl(a1, y)));
            }
            psi[(size_t)jj * nc + col] = y;
            dprev = dj;
            a3prev = a3;
        }
    }
    double2 x = y;
    p[(size_t)(n - 1) * nc + col] = dadd(p[(size_t)(n - 1) * nc + col], x);
    if (FUSE) {
        // v_corr (littleharsh.f90:796-907) in the back sweep: centre j = jp0 + jj takes
        // psi(j); face j takes psi(j+1) - psi(j) (faces jv0+1..jv1-1); ghost/wall rows last
        const size_t ju = (size_t)(d.jp1 - d.ju0);
        u1[ju * nc + col] = dsub(u1[ju * nc + col], dik(dtrk * kxv, x));
        u3[ju * nc + col] = dsub(u3[ju * nc + col], dik(dtrk * kzv, x));
        u1[(ju + 1) * nc + col] = dscl(-g.gwt, u1[ju * nc + col]);
        u3[(ju + 1) * nc + col] = dscl(-g.gwt, u3[ju * nc + col]);
    }
    for (int jj0 = n - 2; jj0 >= 0; jj0 -= CFD_UB) {
        double cc[CFD_UB];
        double2 ya[CFD_UB], pa[CFD_UB], ua[CFD_UB], wa[CFD_UB], va[CFD_UB];
#pragma unroll
        for (int t = 0; t < CFD_UB; ++t)
            if (jj0 - t >= 0) {
                const size_t o = (size_t)(jj0 - t) * nc + col;
                cc[t] = cs[o]; ya[t] = psi[o]; pa[t] = p[o];
                if (FUSE) {
                    const int j = d.jp0 + jj0 - t;
                    ua[t] = u1[(size_t)(j - d.ju0) * nc + col];
                    wa[t] = u3[(size_t)(j - d.ju0) * nc + col];
                    va[t] = u2[(size_t)(j - d.jv0) * nc + col];
                }
            }
#pragma unroll
        for (int t = 0; t < CFD_UB; ++t) {
            if (jj0 - t < 0) break;
            const size_t o = (size_t)(jj0 - t) * nc + col;
            const double2 xp = x;  // psi(j+1)
            x = dsub(ya[t], dscl(cc[t], x));
            if (!FUSE) psi[o] = x;
            p[o] = dadd(pa[t], x);
            if (FUSE) {
                const int j = d.jp0 + jj0 - t;
                u1[(size_t)(j - d.ju0) * nc + col] = dsub(ua[t], dik(dtrk * kxv, x));
                u3[(size_t)(j - d.ju0) * nc + col] = dsub(wa[t], dik(dtrk * kzv, x));
                const size_t jv = (size_t)(j - d.jv0);
                u2[jv * nc + col] = dsub(va[t], dscl(dtrk * g.dthdyv[jv], dsub(xp, x)));
            }
        }
    }
    if (FUSE) {
        u1[col] = dscl(-g.gwb, u1[nc + col]);
        u3[col] = dscl(-g.gwb, u3[nc + col]);
        u2[col] = dc(0, 0);
        u2[(size_t)(d.nyv - 1) * nc + col] = dc(0, 0);
    }
}

// v_corr (littleharsh.f90:796-907) of the stage entry point: u -= dt(a+b) ikx psi, w -= dt(a+b) ikz
// psi, v -= dt(a+b) dthdyv (psi(j+1)-psi(j)), ghost rows by gridweighting, v walls 0; one thread per
// column and a chunk of JC planes.  Its closing divergence follows in k_divergence.  One thread per
// column walking all planes took 366 us at 192 x 193(+90) x 192 FP64, the two launches take 41 + 23.
__global__ void __launch_bounds__(256) k_vcorr_chunk(Dims d, Geo g, double dtrk, double2* __restrict__ u1,
                                                     double2* __restrict__ u2, double2* __restrict__ u3,
                                                     const double2* __restrict__ psi, int JC) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int i = col % d.nkx, q = col / d.nkx;
    const double kxv = g.kx[i], kzv = g.kz[q];
    const size_t nc = d.ncol;
    const int cb = blockIdx.y;
    // u, w at centres j = ju0+1..ju1-1 (= p-points)
    const int jb = d.ju0 + 1 + cb * JC, je = min(jb + JC, d.ju1);
    for (int j = jb; j < je; ++j) {
        const size_t ju = (size_t)(j - d.ju0);
        const double2 ps = psi[(size_t)(j - d.jp0) * nc + col];
        u1[ju * nc + col] = dsub(u1[ju * nc + col], dik(dtrk * kxv, ps));
        u3[ju * nc + col] = dsub(u3[ju * nc + col], dik(dtrk * kzv, ps));
    }
    // v at faces j = jv0+1..jv1-1: psi(j+1) - psi(j)
    const int vb = d.jv0 + 1 + cb * JC, ve = min(vb + JC, d.jv1);
    for (int j = vb; j < ve; ++j) {
        const size_t jv = (size_t)(j - d.jv0);
        const double2 pa = psi[(size_t)(j + 1 - d.jp0) * nc + col], pb = psi[(size_t)(j - d.jp0) * nc + col];
        u2[jv * nc + col] = dsub(u2[jv * nc + col], dscl(dtrk * g.dthdyv[jv], dsub(pa, pb)));
    }
    if (cb == 0) {
        u2[col] = dc(0, 0);
        u2[(size_t)(d.nyv - 1) * nc + col] = dc(0, 0);
        // chunk 0 has just corrected u(ju0+1), the row the bottom ghost extrapolates from
        u1[col] = dscl(-g.gwb, u1[nc + col]);
        u3[col] = dscl(-g.gwb, u3[nc + col]);
    }
    if (je == d.ju1 && jb < je) {
        u1[(size_t)(d.nyu - 1) * nc + col] = dscl(-g.gwt, u1[(size_t)(d.nyu - 2) * nc + col]);
        u3[(size_t)(d.nyu - 1) * nc + col] = dscl(-g.gwt, u3[(size_t)(d.nyu - 2) * nc + col]);
    }
}

// --------------------------------------------------------------------------------------
// Mean mode: flowrate_corr with LUsol0/LU_build0/LU_dec0 (littleharsh.f90:452-484,
// tridLU_3D_IB.f90:320-346, 493-519, 605-622) and flowrateIm (littleharsh.f90:411-430).
// scal[0] = mpgx, scal[1] = Qx, scal[2] = dgx.  The unit-response column spans j = 0..ny (cells
// between the crests plus one each side), as in the reference.  Constant flow rate on columns
// that k_meanflow_warp (colsolve.cuh) holds runs that kernel instead.
// --------------------------------------------------------------------------------------
__global__ void k_meanflow(Dims d, Geo g, double beta, double bdt, double qxt, int ctpress, double2* __restrict__ u1,
                           double* __restrict__ scal, double* __restrict__ work, bool ghosts) {
    // one warp: the flow-rate sums and the final update spread over the lanes (strided
    // reads of the mean-mode column), the tridiagonal solve of the mean mode on lane 0
    if (blockIdx.x != 0) return;
    const int lane = threadIdx.x & 31;
    const int nn = d.ny - 2;
    auto YV = [&](int j) { return g.yv[j - d.jv0]; };
    auto wsum = [](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    double Qx0 = 0.0;
    for (int j = 1 + lane; j <= nn + 1; j += 32) Qx0 += (YV(j) - YV(j - 1)) * u1[(size_t)(j - d.ju0) * d.ncol].x;
    Qx0 = wsum(Qx0);
    if (ctpress == 1) {
        if (lane == 0) scal[1] = Qx0;
        return;
    }
    const int n = nn + 3;
    double* a1 = work;
    double* a2 = work + n;
    double* a3 = work + 2 * n;
    double* x = work + 3 * n;
    for (int j = 1 + lane; j <= nn + 1; j += 32) {
        const int jj = j - d.ju0;
        a1[j] = -beta * g.dyu2i[3 * jj + 0];
        a2[j] = 1.0 - beta * g.dyu2i[3 * jj + 1];
        a3[j] = -beta * g.dyu2i[3 * jj + 2];
    }
    __syncwarp();
    if (lane == 0) {
        a1[0] = 0.0; a2[0] = 1.0; a3[0] = g.gwb;
        a1[nn + 2] = g.gwt; a2[nn + 2] = 1.0; a3[nn + 2] = 0.0;
        a2[0] = 1.0 / a2[0];
        for (int j = 1; j < n; ++j) {
            a3[j - 1] = a3[j - 1] * a2[j - 1];
            a2[j] = 1.0 / (a2[j] - a1[j] * a3[j - 1]);
        }
        x[0] = 0.0 * a2[0];
        for (int j = 1; j < n; ++j) {
            const double rj = (j <= nn + 1) ? bdt : 0.0;
            x[j] = (rj - a1[j] * x[j - 1]) * a2[j];
        }
        for (int j = n - 2; j >= 0; --j) x[j] = x[j] - a3[j] * x[j + 1];
    }
    __syncwarp();
    double Qx1 = 0.0;
    for (int j = 1 + lane; j <= nn + 1; j += 32) Qx1 += (YV(j) - YV(j - 1)) * x[j];
    Qx1 = wsum(Qx1);
    const double gg = (qxt - Qx0) / Qx1;
    if (lane == 0) {
        scal[0] = scal[0] + gg;
        scal[2] = gg;
    }
    for (int j = lane; j <= nn + 2; j += 32) u1[(size_t)(j - d.ju0) * d.ncol].x += gg * x[j];
    if (ghosts) {  // after v_corr: the ghost rows it would have extrapolated
        __syncwarp();
        if (lane == 0) {
            u1[0] = dscl(-g.gwb, u1[d.ncol]);
            u1[(size_t)(d.nyu - 1) * d.ncol] = dscl(-g.gwt, u1[(size_t)(d.nyu - 2) * d.ncol]);
        }
    }
}

// --------------------------------------------------------------------------------------
// Layout conversion f(j,column) <-> [j][column] (32x32 tiles through shared memory).
// --------------------------------------------------------------------------------------
__global__ void k_transpose(const double2* __restrict__ in, double2* __restrict__ out, int rows, int cols,
                            int ldi, int ldo) {
    // in: [rows][cols] with row stride ldi -> out: [cols][rows] with row stride ldo
    __shared__ double2 tile[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int r = by + yy, c = bx + threadIdx.x;
        if (r < rows && c < cols) tile[yy][threadIdx.x] = in[(size_t)r * ldi + c];
    }
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int c = bx + yy, r = by + threadIdx.x;
        if (r < rows && c < cols) out[(size_t)c * ldo + r] = tile[threadIdx.x][yy];
    }
}

// divergence at every p-point (littleharsh.f90:209-244), no state change; one thread per column and
// a chunk of JC planes (blockIdx.y)
__global__ void __launch_bounds__(256) k_divergence(Dims d, Geo g, const double2* __restrict__ u1,
                                                    const double2* __restrict__ u2, const double2* __restrict__ u3,
                                                    double2* __restrict__ divo, int JC) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const double kxv = g.kx[col % d.nkx], kzv = g.kz[col / d.nkx];
    const size_t nc = d.ncol;
    const int j0 = d.jp0 + blockIdx.y * JC;
    for (int j = j0; j <= min(j0 + JC - 1, d.jp1); ++j) {
        const size_t ju = (size_t)(j - d.ju0), jv = (size_t)(j - d.jv0);
        divo[(size_t)(j - d.jp0) * nc + col] =
            dadd(dadd(dik(kxv, u1[ju * nc + col]), dik(kzv, u3[ju * nc + col])),
                 dscl(g.dthdyu[ju], dsub(u2[jv * nc + col], u2[(jv - 1) * nc + col])));
    }
}

// per-block max |z| of a complex array (error(), littleharsh.f90:322-351)
__global__ void k_absmax(const double2* __restrict__ a, size_t n, double* __restrict__ part) {
    __shared__ double sm[256];
    double m = 0.0;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const double2 v = a[t];
        m = nan_max(m, sqrt(v.x * v.x + v.y * v.y));
    }
    sm[threadIdx.x] = m;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sm[threadIdx.x] = nan_max(sm[threadIdx.x], sm[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sm[0];
}

// --------------------------------------------------------------------------------------
// Generic strided transforms with the reference wrapper semantics (cft_buff.f:1-65,
// rft_buff.f:24-86), FP64.  Lines are gathered into shared memory, transformed, scattered.
// grid: x = chunk of CH lines, y = batch (plane) with stride `bstride` doubles.
// --------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_cft_strided(double* __restrict__ c, int ise, int isa, int m, long long bstride,
                                                     FFTDesc fd, const double2* __restrict__ tw_g, int iopt, int CH) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = fd.n;
    double2* buf0 = reinterpret_cast<double2*>(smem_raw);
    double2* buf1 = buf0 + (size_t)n * CH;
    double2* tw = buf1 + (size_t)n * CH;
    double* base = c + (size_t)blockIdx.y * bstride;
    const int l0 = blockIdx.x * CH;
    for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = tw_g[t];
    for (int t = threadIdx.x; t < n * CH; t += blockDim.x) {
        const int b = t % CH, e = t / CH, l = l0 + b;
        buf0[swz(e, b, __ffs(CH) - 1)] =
            l < m ? dc(base[(size_t)l * isa + (size_t)e * ise], base[(size_t)l * isa + (size_t)e * ise + 1]) : dc(0, 0);
    }
    __syncthreads();
    double2* res = fft_lines<double2>(buf0, buf1, CH, fd, tw, iopt < 0 ? -1 : +1);
    const double s = iopt < 0 ? 1.0 / n : 1.0;
    for (int t = threadIdx.x; t < n * CH; t += blockDim.x) {
        const int b = t % CH, e = t / CH, l = l0 + b;
        if (l < m) {
            const double2 v = res[swz(e, b, __ffs(CH) - 1)];
            base[(size_t)l * isa + (size_t)e * ise] = s * v.x;
            base[(size_t)l * isa + (size_t)e * ise + 1] = s * v.y;
        }
    }
}

__global__ void __launch_bounds__(256) k_rft_strided(double* __restrict__ c, int isa, int m, long long bstride,
                                                     FFTDesc fd, const double2* __restrict__ tw_g, int iopt, int CH) {
    // forward: each line a complex transform of length n of (real, 0) data, FFTPACK
    // storage; inverse: two lines per complex transform
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = fd.n;
    double2* buf0 = reinterpret_cast<double2*>(smem_raw);
    double2* buf1 = buf0 + (size_t)n * CH;
    double2* tw = buf1 + (size_t)n * CH;
    double* base = c + (size_t)blockIdx.y * bstride;
    const int l0 = blockIdx.x * CH;
    for (int t = threadIdx.x; t < n; t += blockDim.x) tw[t] = tw_g[t];
    if (iopt > 0) {
        // inverse: CTA line slot b carries the line pair (2(l0+b), 2(l0+b)+1) as one complex
        // transform of X_a + i X_b (both Hermitian extensions of cc(0..n/2), Im cc(0) and
        // Im cc(n/2) ignored), whose output is x_a + i x_b
        for (int t = threadIdx.x; t < n * CH; t += blockDim.x) {
            const int b = t % CH, k = t / CH, la = 2 * (l0 + b), lb = la + 1;
            double2 A = dc(0, 0), B = dc(0, 0);
            const int kk = k <= n / 2 ? k : n - k;
            const bool edge = kk == 0 || kk == n / 2;
            if (la < m) { const double* x = base + (size_t)la * isa; A = dc(x[2 * kk], edge ? 0.0 : x[2 * kk + 1]); }
            if (lb < m) { const double* x = base + (size_t)lb * isa; B = dc(x[2 * kk], edge ? 0.0 : x[2 * kk + 1]); }
            if (k > n / 2) { A.y = -A.y; B.y = -B.y; }
            buf0[swz(k, b, __ffs(CH) - 1)] = dc(A.x - B.y, A.y + B.x);
        }
        __syncthreads();
        double2* res = fft_lines<double2>(buf0, buf1, CH, fd, tw, +1);
        for (int t = threadIdx.x; t < n * CH; t += blockDim.x) {
            const int b = t % CH, e = t / CH, la = 2 * (l0 + b), lb = la + 1;
            const double2 v = res[swz(e, b, __ffs(CH) - 1)];
            if (la < m) base[(size_t)la * isa + e] = v.x;
            if (lb < m) base[(size_t)lb * isa + e] = v.y;
        }
        return;
    }
    for (int t = threadIdx.x; t < n * CH; t += blockDim.x) {
        const int b = t % CH, k = t / CH, l = l0 + b;
        double2 v = dc(0, 0);
        if (l < m) v = dc(base[(size_t)l * isa + k], 0.0);
        buf0[swz(k, b, __ffs(CH) - 1)] = v;
    }
    __syncthreads();
    double2* res = fft_lines<double2>(buf0, buf1, CH, fd, tw, -1);
    for (int t = threadIdx.x; t < (n + 2) * CH; t += blockDim.x) {
        const int b = t % CH, e = t / CH, l = l0 + b;
        if (l >= m) continue;
        double* x = base + (size_t)l * isa;
        const int k = e >> 1;
        const double2 v = res[swz(k, b, __ffs(CH) - 1)];
        double val = (e & 1) ? v.y : v.x;
        if ((e & 1) && (k == 0 || k == n / 2)) val = 0.0;
        x[e] = val / n;
    }
}

}  // namespace cfd
