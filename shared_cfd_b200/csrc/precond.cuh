// precond.cuh -- the cell phase of the preconditioned schemes' residual, shared by the
// generic and the fused residual kernels.
#pragma once

#include "scfd_internal.h"

namespace scfd {

// From the cell's right-hand side R: Dq, and the coefficients the sweeps read.  D: dimq, a
// constant where the species count is one.
//
// RES_DUAL: set_ABpm of the preconditioned dual time (dual/2d/sch_dual.raw.f90:38-83):
// low-Mach reference velocity, preconditioned spectral radii, pseudo time step from
// cfl_tau, and the scalars of Gamma^-1, S, S^-1; Dq = R - Vol dqdt, then
// Dq += pre_sca(2) (pre2 . Dq) pre1 (time_dual_viscous.f90:29), pre1 = (Y, u, v, H),
// pre2 = (g1 Vs/2 + DHi, -g1 u, -g1 v, g1).
// RES_PRECON, RES_PRECON_LUSGS: set_ABpm of time_scheme/precon/2d (sch_precon.raw.f90:28-77,
// 194-197): the same velocity and radii, the local time step (written to dt_mat:
// set_dqdt and alpha use it), phh of pre1 = phh (Y, u, v, H); then
// Dq = R + pre1 (pre2 . R) [- Vol dqdt] (time_precon_viscous.f90:18-27).
template <int MODE>
__device__ __forceinline__ void precond_cell(const View& v, int p, int i, int j, long long c, int D, const double* R,
                                             double vol, double dtl, bool first) {
    const long long N = v.ncell;
    const int nY = D - 3;
    const double rho = v.w[c], u = v.w[N + c], vv = v.w[2 * N + c], pr = v.w[3 * N + c];
    const double gamm = v.w[(D + 1) * N + c], H = v.w[(D + 2) * N + c];
    const double mu = v.w[(D + 4) * N + c], dsa = v.dsci[c], dsb = v.dscj[c];
    const double cs = sqrt(gamm * pr / rho);
    const double unA = v.vnci[c] * u + v.vnci[N + c] * vv;
    const double unB = v.vncj[c] * u + v.vncj[N + c] * vv;
    const double Vs = u * u + vv * vv;
    const double Vv = mu / rho / fmin(dsa, dsb);
    const double Ur = fmin(fmax(Vv, sqrt(Vs)), cs);
    const double phi = 1.0 / (Ur * Ur) - 1.0 / (cs * cs);
    const double alp = 0.5 * (1.0 - (Ur / cs) * (Ur / cs));
    double ud = unA * (1.0 - alp), cd = sqrt(alp * alp * (unA * unA) + Ur * Ur);
    const double nuA = fabs(ud) + cd;
    ud = unB * (1.0 - alp);
    cd = sqrt(alp * alp * (unB * unB) + Ur * Ur);
    const double nuB = fabs(ud) + cd;
    const long long cim = cidx(v.P, p, i - 1, j), cjm = cidx(v.P, p, i, j - 1);
    const double uds = nuA * (v.dsi[c] + v.dsi[cim]) + nuB * (v.dsj[c] + v.dsj[cjm]);
    const double g1 = gamm - 1.0;
    v.nuA[c] = nuA;
    v.nuB[c] = nuB;
    auto dqdt = [&](int k, double dt) {
        const double qk = v.q[k * N + c], qpk = v.qp[k * N + c];
        return first ? (qk - qpk) / dt : (3.0 * qk - 4.0 * qpk + v.qpp[k * N + c]) / (2.0 * dt);
    };
    auto pre2 = [&](int k) {
        return k < nY ? 0.5 * g1 * Vs + v.DHi[k * N + c] : (k == nY ? -g1 * u : (k == nY + 1 ? -g1 * vv : g1));
    };
    auto pre1 = [&](int k) { return k < nY ? v.w[(4 + k) * N + c] : (k == nY ? u : (k == nY + 1 ? vv : H)); };
    if (MODE == RES_DUAL) {
        const double dtau = v.cfl_tau * vol / fmax(uds, mu / rho);
        const double al = 1.0 / (vol / dtau + dsa * nuA + dsb * nuB);
        const double beta = 3.0 * vol / (2.0 * dtl) * al;
        const double c2 = cs * cs;
        const double s2 = -1.0 / (1.0 / phi + c2);
        v.alpha[c] = al;
        v.pre[c] = 1.0 + beta;
        v.pre[N + c] = s2;
        v.pre[2 * N + c] = -1.0 / (1.0 / phi + c2) / (1.0 / beta + 1.0);
        v.pre[3 * N + c] = beta / ((1.0 + beta) / phi + c2);
        double t = 0.0;
        for (int k = 0; k < D; ++k) t = t + pre2(k) * (R[k] - vol * dqdt(k, dtl));
        for (int k = 0; k < D; ++k) {
            const double rhs = R[k] - vol * dqdt(k, dtl);
            v.Dq[k * N + c] = rhs + s2 * t * pre1(k);
        }
        return;
    }
    const double dt = v.cfl * vol / fmax(uds, mu / rho);
    v.dt_mat[c] = dt;
    const double phh = -1.0 / (cs * cs + 1.0 / phi);
    const double tmp = MODE == RES_PRECON ? 3.0 * vol / (2.0 * dt) + dsa * nuA + dsb * nuB
                                          : vol / dt + dsa * nuA + dsb * nuB;
    v.alpha[c] = 1.0 / tmp;
    v.pre[c] = phh;
    double t = 0.0;
    for (int k = 0; k < D; ++k) t = t + pre2(k) * R[k];
    for (int k = 0; k < D; ++k) {
        double rhs = R[k] + phh * pre1(k) * t;
        if (MODE == RES_PRECON) rhs = rhs - vol * dqdt(k, dt);
        v.Dq[k * N + c] = rhs;
    }
}

}  // namespace scfd
