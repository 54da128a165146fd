// cell_ops.cuh -- per-cell pieces of set_dt and set_BC that more than one kernel runs.
#pragma once

#include "scfd_internal.h"

namespace scfd {

// the time step of one cell (store/time_step/{global,local}/set_dt.f90), from its w
__device__ __forceinline__ double cell_dt(const View& v, int p, int i, int j) {
    const long long N = v.ncell;
    const long long c = cidx(v.P, p, i, j);
    const long long cim = cidx(v.P, p, i - 1, j), cjm = cidx(v.P, p, i, j - 1);
    const double rho = v.w[c], u = v.w[N + c], vv = v.w[2 * N + c], pr = v.w[3 * N + c];
    const double a = sqrt(v.w[(v.D + 1) * N + c] * pr / rho);
    double uds = 0.0, un;
    un = v.vni[c] * u + v.vni[N + c] * vv;
    uds = uds + (fabs(un) + a) * v.dsi[c];
    un = v.vni[cim] * u + v.vni[N + cim] * vv;
    uds = uds + (fabs(un) + a) * v.dsi[cim];
    un = v.vnj[c] * u + v.vnj[N + c] * vv;
    uds = uds + (fabs(un) + a) * v.dsj[c];
    un = v.vnj[cjm] * u + v.vnj[N + cjm] * vv;
    uds = uds + (fabs(un) + a) * v.dsj[cjm];
    return v.cfl * v.Vol[c] / fmax(uds, v.w[(v.D + 4) * N + c] / rho);
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
