// cell_ops.cuh -- per-cell pieces of set_dt and set_BC that more than one kernel runs.
#pragma once

#include "scfd_internal.h"

namespace scfd {

// What set_dt reads of a cell besides its state: loaded ahead of the state where that is
// still being computed.
struct DtMetrics {
    double ni1, ni2, dsi, mi1, mi2, dsim, nj1, nj2, dsj, mj1, mj2, dsjm, vol;
    __device__ __forceinline__ DtMetrics(const View& v, int p, int i, int j) {
        const long long N = v.ncell;
        const long long c = cidx(v.P, p, i, j), cim = cidx(v.P, p, i - 1, j), cjm = cidx(v.P, p, i, j - 1);
        ni1 = v.vni[c], ni2 = v.vni[N + c], dsi = v.dsi[c];
        mi1 = v.vni[cim], mi2 = v.vni[N + cim], dsim = v.dsi[cim];
        nj1 = v.vnj[c], nj2 = v.vnj[N + c], dsj = v.dsj[c];
        mj1 = v.vnj[cjm], mj2 = v.vnj[N + cjm], dsjm = v.dsj[cjm];
        vol = v.Vol[c];
    }
};
// the time step of one cell (store/time_step/{global,local}/set_dt.f90)
__device__ __forceinline__ double cell_dt(const View& v, const DtMetrics& m, double rho, double u, double vv, double pr,
                                          double gamma, double mu) {
    const double a = sqrt(gamma * pr / rho);
    double uds = 0.0, un;
    un = m.ni1 * u + m.ni2 * vv;
    uds = uds + (fabs(un) + a) * m.dsi;
    un = m.mi1 * u + m.mi2 * vv;
    uds = uds + (fabs(un) + a) * m.dsim;
    un = m.nj1 * u + m.nj2 * vv;
    uds = uds + (fabs(un) + a) * m.dsj;
    un = m.mj1 * u + m.mj2 * vv;
    uds = uds + (fabs(un) + a) * m.dsjm;
    return v.cfl * m.vol / fmax(uds, mu / rho);
}
// the same from w
__device__ __forceinline__ double cell_dt(const View& v, int p, int i, int j) {
    const long long N = v.ncell, c = cidx(v.P, p, i, j);
    return cell_dt(v, DtMetrics(v, p, i, j), v.w[c], v.w[N + c], v.w[2 * N + c], v.w[3 * N + c], v.w[(v.D + 1) * N + c],
                   v.w[(v.D + 4) * N + c]);
}

// dt_grbl and tt (global: tt = tt + dt_grbl, set_dt.f90:40-42; fixed dt likewise); one thread.
// The minimum starts again for the next step.
__device__ __forceinline__ void dt_final(const View& v) {
    if (v.dt_mode == SCFD_DT_GLOBAL) {
        v.sc->dt_grbl = __longlong_as_double((long long)v.sc->dtmin_bits);
        v.sc->tt = v.sc->tt + v.sc->dt_grbl;
        v.sc->dtmin_bits = kDtInf;
    } else if (v.dt_mode == SCFD_DT_FIXED) {
        v.sc->dt_grbl = v.dt_fixed;
        v.sc->tt = v.sc->tt + v.sc->dt_grbl;
    }
}

}  // namespace scfd
