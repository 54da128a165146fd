// k_bc.cu -- set_BC on the device.
//
// The reference fills ghost cells in this order (store/cond/no-nV/condition.tail.f90
// and the generated condition.f90): section_exchange (block-interface halo,
// lines 2-70) -> user i-boundaries -> user j-boundaries -> set_corners
// (lines 331-356).  Every ghost write of the first three phases reads only
// interior cells, so the host expands them into one list of ghost-cell
// operations, keeps the last writer of each ghost cell in reference order, and
// a single launch applies them all.  set_corners reads ghost cells: the same launch
// forms the values it reads from their own operations instead of waiting for them.
#include "cell_ops.cuh"

namespace scfd {

// component m (m < W of w, then vhi) of the ghost cell that op writes
__device__ __forceinline__ double ghost_value(const View& v, const GhostOp& op, const double* bcval, int valstride, int m) {
    const int W = v.W, nY = v.nY;
    const long long N = v.ncell, s = op.src;
    const double* val = bcval + (long long)op.bc * valstride;
    const double* w = v.w;
    if (m >= W)  // vhi
        return op.kind == SCFD_BC_FIXED || op.kind == SCFD_BC_FIXED_PIN ? val[m] : v.vhi[(m - W) * N + s];
    switch (op.kind) {
        case SCFD_BC_FIXED: return val[m];
        case SCFD_BC_FIXED_PIN: {
            const double pin = w[3 * N + s];
            return m == 0 ? pin * val[W + nY] / val[W + nY + 1] : (m == 3 ? pin : val[m]);
        }
        case SCFD_BC_OUTFLOW_P: return m == 3 ? val[0] : w[m * N + s];
        case SCFD_BC_SLIP:
            if (m == 1 || m == 2) {
                const double u = w[N + s], vv = w[2 * N + s];
                const double un = u * op.n1 + vv * op.n2;
                return m == 1 ? u - 2.0 * un * op.n1 : vv - 2.0 * un * op.n2;
            }
            return w[m * N + s];
        case SCFD_BC_NOSLIP: return (m == 1 || m == 2) ? val[m - 1] * 2.0 - w[m * N + s] : w[m * N + s];
        default: return w[m * N + s];
    }
}

// One thread per (ghost op, component), then per (corner, component): component m < W of
// w, then vhi (condition.tail.f90:331-356 for the corners).
__global__ void k_ghost(View v, const GhostOp* ops, int nops, const CornerOp* corners, int ncorners, const double* bcval,
                        int valstride) {
    const int W = v.W, NC = W + v.nY;
    const long long N = v.ncell;
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < (long long)nops * NC) {
        const int m = (int)(t / nops), o = (int)(t - (long long)m * nops);
        const GhostOp op = ops[o];
        double* f = m < W ? v.w + m * N : v.vhi + (m - W) * N;
        f[op.dst] = ghost_value(v, op, bcval, valstride, m);
        return;
    }
    t -= (long long)nops * NC;
    if (t >= (long long)ncorners * NC) return;
    const int m = (int)(t % NC);
    const CornerOp co = corners[t / NC];
    double* f = m < W ? v.w + m * N : v.vhi + (m - W) * N;
    const double b = co.ob >= 0 ? ghost_value(v, ops[co.ob], bcval, valstride, m) : f[co.b];
    const double c = co.oc >= 0 ? ghost_value(v, ops[co.oc], bcval, valstride, m) : f[co.c];
    f[co.dst] = 1.0 / 3.0 * (f[co.a] + b + c);
}

// the ghost-cell writes without set_corners (for stencils that never read corners)
int launch_ghost_ops(const View& v, cudaStream_t s, const GhostOp* ops, int nops, const double* bcval, int valstride) {
    return launch_ghosts(v, s, ops, nops, nullptr, 0, bcval, valstride);
}

int launch_ghosts(const View& v, cudaStream_t s, const GhostOp* ops, int nops, const CornerOp* corners, int ncorners,
                  const double* bcval, int valstride) {
    const long long nt = ((long long)nops + ncorners) * (v.W + v.nY);
    if (nt <= 0) return 0;
    k_ghost<<<(unsigned)((nt + 255) / 256), 256, 0, s>>>(v, ops, nops, corners, ncorners, bcval, valstride);
    return 1;
}

}  // namespace scfd
