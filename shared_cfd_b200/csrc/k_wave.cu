// k_wave.cu -- LU-SGS sweeps as cluster wavefronts.
//
// Restates calc_next_step_implicit of store/time_scheme/LU-SGS/{2d,q2d}/time_lusgs_viscous.f90,
// NR/{2d,q2d}/time_NR_viscous.f90:30-108, dual/2d/time_dual_viscous.f90:30-125 and
// precon/2d/time_precon_viscous.f90 with the split Jacobians of set_ABpm
// (sch_lusgs.raw.f90:1-141, NR/q2d/sch_NR.raw.f90:1-149), applied matrix-free.
//
// Schedule.  A strip is 8 rows of one plane, swept by one warp with four lanes
// per cell; row l of the strip at sweep step t updates column t - l (the
// hyperplane order i + j of the reference, row l lagging row l - 1 by one
// step).  The i - 1 neighbour's product is in the lane's registers, the j - 1
// neighbour's arrives from the row below by __shfl_up, and the bottom row of a
// strip takes the top row of the strip below through a hand-off ring in shared
// memory.
//
// What bounds it: the chain of ni + nj dependent steps, and in each step the
// issue and the dependence chain of one warp (about 2 cycles per FP64 or FP32
// instruction, 4 per shuffle), not memory (786 k cells of 9 species FP64: 342 MB in
// 269 us, 1.27 TB/s, 19 % of the copy rate).  So a cell's D components
// are spread over four lanes, a plane's rows over all the SMs that the clusters
// can have, and what is not the chain is taken off the step: the next step's
// record is read into registers while this one is computed, results go straight to
// global memory (nothing waits for them), and record loads, the release of
// consumed hand-off chunks and the hand-off itself have warps of their own.
// Measured (B200, per launch, forward / backward): 786 k cells of 9 species FP64
// 269 / 254 us, FP32 200 / 197 us, against 426 / 414 and 289 / 288 us for 32-row
// strips with one lane per cell; 256 x 128 cells of one species FP64 70 / 68 us
// against 103 / 101 us.  A step takes 190-196 (forward) and 185 ns (backward) FP64 and
// 140 ns FP32 at 9 species, 135 and 98 ns at one (one lane per cell: 398, 255, 248 and
// 180 ns), of which the hand-off is about 10.
//
// A task is 256 consecutive rows of one plane at most, run by one thread-block
// cluster of 16 CTAs with two strips each (128 rows and 8 CTAs, the largest portable
// cluster, on a device or part of one that holds none of 16: its plane's top rows then
// travel through global memory twice as often).  A strip's top row is staged in its
// CTA's shared memory; every HK columns one bulk copy moves the chunk into the
// next CTA's hand-off ring (distributed shared memory), completing a transaction count on
// an mbarrier of the receiver, which releases consumed chunks with a remote arrive.  From a
// CTA's first strip to its second the top row is written into the ring directly.  A task with a successor holds
// all its strips, so only the last strip of a cluster ever publishes to global
// memory and the others only to the next strip.  Between tasks of one plane the
// top row travels through global memory: a warp of the last CTA copies it
// out and publishes a progress counter (release; several chunks at once when they
// are ready, since the fence takes longer than a chunk), a warp of the next task's
// rank 0 polls it (acquire) and bulk-copies the chunks into its own ring.
// Tasks are taken from a ticket counter in dependency order, so a cluster only
// ever waits for tasks that are already running.
//
// Warps of a CTA: 0, 1 compute the two strips (the wavefront only); 2, 3 stream
// their records through a ring of slots (bulk copies completing on mbarriers) and
// release hand-off chunks; 6, 7 pass their top rows on; 4 fetches the chunks of
// the task below.  Every wait is bounded; a wait that gives up sets SCFD_E_SPIN
// and the kernel winds down instead of hanging.
//
// Records (k_pack, in the cell order of the sweep), for the cell
// (i = t - l + 1, j = R s + 1 + l) and lane = 4 l + sub:
//   X[strip][step t][slot][lane]     x: the right-hand side (WL::SCALED: times
//                                    alpha), then the forward result, then Dq
//   C[strip][step t]: the lane's own coefficients [group][lane][GP] (WL), then the
//                     fields its four lanes share, [group][row][GM] (CM9, CM1)
// The backward sweep walks the same records with steps and rows reversed.
// k_unpack applies q += omega Dq back in the cell layout.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>

#include "async_ptx.h"
#include "scfd_internal.h"

namespace scfd {

using namespace ptx;

namespace {

constexpr int LPC = 4;   // lanes per cell
constexpr int R = 32 / LPC;  // rows per strip
constexpr int UPC = 2;   // strips per CTA
constexpr int HK = 4;    // hand-off columns per chunk
constexpr int HS = 32;   // hand-off ring chunks
constexpr int SPB = 8;   // steps per record slot (one wait and one release each)
constexpr int kPadSteps = 8;  // zero step blocks before and after each strip's records
constexpr int kThreads = 256; // of a sweep CTA
// warps by role: 0, 1 compute (on sub-partitions 0 and 1); the record loads and the
// hand-off wait on sub-partitions 2 and 3, away from them
constexpr int kWarpLoad = 2, kWarpIn = 4, kWarpOut = 6;
constexpr long long kSpin = 1ll << 22;   // polls of a wait
constexpr long long kDrain = 1ll << 17;  // cycles (70 us)

// hand-off chunks of a strip's top row for a plane of ni columns: chunk j
// holds the columns 4j-3 .. 4j (HK = 4), j = 0 .. (ni + 2) / 4
__host__ __device__ constexpr int chunks_of(int ni) { return (ni + 2) / 4 + 1; }

template <typename T, int G>
struct VecOf;
template <>
struct VecOf<float, 4> {
    using type = float4;
};
template <>
struct VecOf<float, 2> {
    using type = float2;
};
template <>
struct VecOf<double, 2> {
    using type = double2;
};

// The fields of a cell that its lanes share (set_ABpm's quantities,
// sch_lusgs.raw.f90:27-50,134-136; NR/q2d/sch_NR.raw.f90:43-50,143-144), formed in
// FP64 by k_pack.  Fields both sweeps read come first, then the forward sweep's,
// then the backward sweep's, each a whole number of 16-byte vectors:
//   AL            alpha = 1/(Vol/dt + dsci nuA + dscj nuB)   (NR: 3 Vol/(2 dt))
//   DV            -g1 v, dpdq of rho v
//   per direction (A: i, ds = dsci, n = vnci; B: j, ds = dscj, n = vncj), with
//   fa = ds/2, un = n.u and nu = |un| + sound speed:
//   P1 = fa n1, P2 = fa n2, PU = fa un, LP = fa (un + nu), LM = fa (un - nu)
//   AA, RQ        alpha*Area and 1/(1 - alpha*Area*dpdq_my)  (q2d pressure source; 0 and 1 in 2d)
// 8 or 9 species: a lane holds three components (three species, or rho u, rho v,
// rho E), its own coefficients are their (dpdq, primitive vector) pairs.
struct CM9 {
    static constexpr int AL = 0, DV = 1, P1A = 2, P2A = 3, PUA = 4, PUB = 5, P1B = 6, P2B = 7, LPA = 8, LPB = 9,
                         AA = 10, RQ = 11, LMA = 12, LMB = 13;
    static constexpr int FWD = 8, BWD = 12, BWD_END = 14, PRE = 16, END = 16;  // first fields of the parts
};
// One species: a lane holds one component and forms P, S and the directions'
// products from all four; its own coefficients are (primitive, pA, pB), p the
// factor of P in its product.  dpdq is shared: D0 (species), DU, DV, DE.
// The preconditioned schemes (dual/2d/sch_dual.raw.f90:38-83, precon/2d/sch_precon.raw.f90:28-77;
// nu is then the preconditioned radius) add
//   K1, S2        1 + s2 p2.p1 and s2: the split Jacobians are (I + s2 p1 p2^T)
//                 (n1 A + n2 B)/2 +- nu/2 with p1 = (Y, u, v, H), p2 = dpdq
//   S1, S3, S4, I1  dual's S: x -> s1 (x + s3 (p2.x) p1), S^-1: x -> (x + s4 (p2.x) p1) / s1
//   Y0, U, V, H   p1
struct CM1 {
    static constexpr int AL = 0, D0 = 1, DU = 2, DE = 3, DV = 4, P1A = 5, P2A = 6, PUA = 7, PUB = 8, P1B = 9, P2B = 10,
                         K1 = 11, LPA = 12, LPB = 13, AA = 14, RQ = 15, LMA = 16, LMB = 17, S1 = 18, S3 = 19, S2 = 20,
                         S4 = 21, I1 = 22, Y0 = 23, U = 24, V = 25, H = 26;
    static constexpr int FWD = 12, BWD = 16, BWD_END = 20, PRE = 20, END = 28;
};

// PRE: 0 LU-SGS and NR, 1 the preconditioned schemes (one species)
template <typename RT, int NY_, int PRE_>
struct WL {
    static constexpr int NY = NY_, PRE = PRE_;
    using CM = typename std::conditional<NY == 1, CM1, CM9>::type;
    static constexpr int D = NY + 3;
    static constexpr int K = NY == 1 ? 1 : 3;                 // component slots per lane
    static constexpr int GM = 16 / (int)sizeof(RT);           // shared fields per vector
    static constexpr int GP = NY == 1 ? GM : 2;               // own coefficients per vector
    static constexpr int NP = (NY == 1 ? 4 : 2 * K) / GP;     // own vectors
    static constexpr int NM = (PRE ? CM::END : CM::PRE) / GM; // shared vectors
    static constexpr int XS = K * 32;                         // elements of one step block of X
    static constexpr int CO = NP * 32 * GP;                   // shared fields' offset in a step block of C
    static constexpr int CS = CO + NM * R * GM;
    static constexpr int D4 = LPC * K;                        // hand-off column
    static constexpr bool SCALED = NY != 1 || PRE != 0;       // the right-hand side in X carries alpha
    // slots in the ring: as many as shared memory takes, 3 for FP64 (24 steps of
    // 3.3 KB at 9 species for each of two strips), 4 for FP32
    static constexpr int PFB = sizeof(RT) == 8 ? 3 : 4;
    static constexpr int NBAR = 2 * PFB + 4 * HS;
    static constexpr size_t UNIT = sizeof(RT) * ((size_t)PFB * SPB * (XS + CS) + 2 * HS * HK * D4) + 8 * NBAR;
    static constexpr size_t SMEM = UPC * UNIT + 16;
    static_assert(NY == 1 || NY == 8 || NY == 9, "components fit the lanes' slots");
    static_assert(UNIT % 16 == 0, "the second strip's rings are 16-byte aligned");
    // arrivals of a phase of barrier k of the CTA's strip n, in the order of Unit: rfull, rdone,
    // xfull, pempty, hempty, oful.  The top row's four lanes arrive on its own chunks (oful),
    // and the first strip's on those that it writes into the second's ring (xfull).
    static __host__ __device__ constexpr int arrivals(int n, int k) {
        const int c = (k - 2 * PFB) / HS;
        return k >= 2 * PFB && (c == 3 || (c == 0 && n == 1)) ? LPC : 1;
    }
    // the component in slot s of lane sub, -1: none (a zero slot)
    static __host__ __device__ constexpr int comp(int sub, int s) {
        return NY == 1 ? sub : sub == 3 ? NY + s : 3 * sub + s < NY ? 3 * sub + s : -1;
    }
};

}  // namespace

// ---------------------------------------------------------------------------
// k_pack: cell layout -> records (32 steps x R rows of one strip per block).
// Cells are read along i (thread: step x, row y), up to 16 fields at a time go
// through shared memory, and a warp writes a step's block (lane = 4 row + sub) as
// whole lines.  Block 0 also resets the sweeps' counters.
// ---------------------------------------------------------------------------
template <typename T, int NY, int PRE>
__global__ void __launch_bounds__(32 * R, 2)
k_pack(View v, const int2* blk, const int4* strips, const long long* step_off, T* X, T* Cr, int nr_mode, int* progress,
       int nprogress, int* tickets) {
    using L = WL<T, NY, PRE>;
    using CM = typename L::CM;
    constexpr int D = NY + 3, K = L::K, GM = L::GM, NM = L::NM;
    constexpr int NT = 16;  // fields per pass
    __shared__ T tile[NT][R][33];
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if (blockIdx.x == 0) {
        for (int k = tid; k < nprogress; k += 32 * R) progress[k] = 0;
        if (tid < 3) tickets[tid] = 0;
    }
    const int2 b = blk[blockIdx.x];
    const int4 st = strips[b.x];
    const int p = st.x, s = st.y;
    const int ni = v.P.ni[p], nj = v.P.nj[p];
    const int tt = threadIdx.x, l = threadIdx.y;
    const int t = b.y + tt;
    const int cc = t - l;
    const int i = cc + 1, j = R * s + 1 + l;
    const bool ok = cc >= 0 && cc < ni && j <= nj && t < ni + R - 1;
    const long long N = v.ncell;
    const long long c = ok ? cidx(v.P, p, i, j) : 0;
    // all of the cell's values before the first barrier, so that their loads overlap (read
    // pass by pass they took a load latency each: 14.5 us for 768 cells)
    double xq[D], dh[NY], yy[NY];
#pragma unroll
    for (int k = 0; k < D; ++k) xq[k] = ok ? v.Dq[k * N + c] : 0.0;
#pragma unroll
    for (int k = 0; k < NY; ++k) {
        dh[k] = ok ? v.DHi[k * N + c] : 0.0;
        yy[k] = ok ? v.w[(4 + k) * N + c] : 0.0;
    }
    double cm[NM * GM] = {};  // shared fields
    double u = 0.0, vv = 0.0, H = 0.0, g1 = 0.0, hvs = 0.0, al = 0.0;
    if (ok) {
        const double* w = v.w;
        const double rho = w[c];
        const double pr = w[3 * N + c];
        u = w[N + c];
        vv = w[2 * N + c];
        H = w[(D + 2) * N + c];
        const double gamm = w[(D + 1) * N + c];
        g1 = gamm - 1.0;
        hvs = 0.5 * g1 * (u * u + vv * vv);
        const double cs = sqrt(gamm * pr / rho);
        const double dsa = v.dsci[c], dsb = v.dscj[c], vol = v.Vol[c];
        double nus[2];
        for (int d = 0; d < 2; ++d) {
            const double fa = 0.5 * (d == 0 ? dsa : dsb);
            const double n1 = d == 0 ? v.vnci[c] : v.vncj[c], n2 = d == 0 ? v.vnci[N + c] : v.vncj[N + c];
            const double un = n1 * u + n2 * vv;
            const double nu = PRE ? (d == 0 ? v.nuA[c] : v.nuB[c]) : fabs(un) + cs;
            nus[d] = nu;
            cm[d == 0 ? CM::P1A : CM::P1B] = fa * n1;
            cm[d == 0 ? CM::P2A : CM::P2B] = fa * n2;
            cm[d == 0 ? CM::PUA : CM::PUB] = fa * un;
            cm[d == 0 ? CM::LPA : CM::LPB] = fa * (un + nu);
            cm[d == 0 ? CM::LMA : CM::LMB] = fa * (un - nu);
        }
        if (PRE) {
            al = v.alpha[c];
        } else {
            const double dtl = v.dt_mode == SCFD_DT_LOCAL ? v.dt_mat[c] : v.sc->dt_grbl;
            const double tmp = nr_mode ? 3.0 * vol / (2.0 * dtl) + dsa * nus[0] + dsb * nus[1]
                                       : vol / dtl + dsa * nus[0] + dsb * nus[1];
            al = 1.0 / tmp;
        }
        cm[CM::AL] = al;
        cm[CM::DV] = -g1 * vv;
        cm[CM::RQ] = 1.0;
        if (v.dim == SCFD_DIM_Q2D) {
            const double aA = al * v.Area[c];
            cm[CM::AA] = aA;
            cm[CM::RQ] = 1.0 / (1.0 - aA * (-g1 * vv));
        }
        if constexpr (NY == 1) {
            cm[CM::D0] = hvs + dh[0];
            cm[CM::DU] = -g1 * u;
            cm[CM::DE] = g1;
            if constexpr (PRE != 0) {
                const bool dual = v.scheme == SCFD_SCHEME_DUAL;
                const double s2 = dual ? v.pre[N + c] : v.pre[c];
                // p2 . p1
                const double k0 = (hvs + dh[0]) * yy[0] + g1 * (H - (u * u + vv * vv));
                cm[CM::K1] = 1.0 + s2 * k0;
                cm[CM::S2] = s2;
                cm[CM::S1] = dual ? v.pre[c] : 1.0;
                cm[CM::S3] = dual ? v.pre[2 * N + c] : 0.0;
                cm[CM::S4] = dual ? v.pre[3 * N + c] : 0.0;
                cm[CM::I1] = dual ? 1.0 / v.pre[c] : 1.0;
                cm[CM::Y0] = yy[0];
                cm[CM::U] = u;
                cm[CM::V] = vv;
                cm[CM::H] = H;
            }
        }
    }
    auto xval = [&](int k) -> double {
        return k < 0 ? 0.0 : L::SCALED ? al * xq[k < 0 ? 0 : k] : xq[k < 0 ? 0 : k];
    };
    auto dpdq = [&](int k) -> double {
        return k < 0 ? 0.0 : k < NY ? hvs + dh[k < 0 || k >= NY ? 0 : k] : k == NY ? -g1 * u : k == NY + 1 ? 0.0 : g1;
    };
    auto prim = [&](int k) -> double {
        return k < 0 ? 0.0 : k < NY ? yy[k < 0 || k >= NY ? 0 : k] : k == NY ? u : k == NY + 1 ? vv : H;
    };
    // own coefficient e of (sub, slot): NY = 1 (primitive, pA, pB, 0), else (dpdq, primitive); dpdq of
    // rho v is left to the shared DV, which follows the pressure source
    auto own = [&](int sub, int sl, int e) -> double {
        const int k = L::comp(sub, sl);
        if constexpr (NY == 1) {
            if (e == 0) return prim(k);
            if (e == 1) return k == 1 ? cm[CM::P1A] : k == 2 ? cm[CM::P2A] : k == 3 ? cm[CM::PUA] : 0.0;
            if (e == 2) return k == 1 ? cm[CM::P1B] : k == 2 ? cm[CM::P2B] : k == 3 ? cm[CM::PUB] : 0.0;
            return 0.0;
        } else {
            return e == 0 ? dpdq(k) : prim(k);
        }
    };
    const long long s0 = step_off[b.x] + kPadSteps + b.y;
    T* outX = X + s0 * L::XS;
    T* outC = Cr + s0 * L::CS;
    const int nt = min(32, ni + R - 1 - b.y);
    const int ln = threadIdx.x, lrow = ln / LPC, lsub = ln % LPC;
    // x
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int q = 0; q < LPC; ++q) tile[k * LPC + q][l][tt] = T(xval(L::comp(q, k)));
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int wt = threadIdx.y + r * R;
        if (wt < nt) {
#pragma unroll
            for (int k = 0; k < K; ++k) outX[(long long)wt * L::XS + k * 32 + ln] = tile[k * LPC + lsub][lrow][wt];
        }
    }
    // the lanes' own coefficients: EP per lane and slot, slots in pairs
    constexpr int EP = NY == 1 ? 4 : 2;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 2) {
        __syncthreads();
#pragma unroll
        for (int k = k0; k < k0 + 2 && k < K; ++k)
#pragma unroll
            for (int q = 0; q < LPC; ++q)
#pragma unroll
                for (int e = 0; e < EP; ++e) tile[((k - k0) * LPC + q) * EP + e][l][tt] = T(own(q, k, e));
        __syncthreads();
        using VP = typename VecOf<T, L::GP>::type;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int wt = threadIdx.y + r * R;
            if (wt < nt) {
                T* dst = outC + (long long)wt * L::CS;
#pragma unroll
                for (int k = k0; k < k0 + 2 && k < K; ++k)
#pragma unroll
                    for (int g = 0; g < EP / L::GP; ++g) {
                        T z[L::GP];
#pragma unroll
                        for (int e = 0; e < L::GP; ++e) z[e] = tile[((k - k0) * LPC + lsub) * EP + g * L::GP + e][lrow][wt];
                        *reinterpret_cast<VP*>(dst + ((k * EP / L::GP + g) * 32 + ln) * L::GP) = *reinterpret_cast<VP*>(z);
                    }
            }
        }
    }
    // the shared fields
    using VM = typename VecOf<T, GM>::type;
#pragma unroll
    for (int f0 = 0; f0 < NM * GM; f0 += NT) {
        __syncthreads();
#pragma unroll
        for (int f = f0; f < f0 + NT && f < NM * GM; ++f) tile[f - f0][l][tt] = T(cm[f]);
        __syncthreads();
        constexpr int GR = 32 / R;  // vectors per warp pass
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int wt = threadIdx.y + r * R;
            if (wt < nt) {
#pragma unroll
                for (int g0 = 0; g0 < NT / GM; g0 += GR) {
                    const int g = g0 + ln / R, row = ln % R;
                    if (f0 / GM + g < NM && g < NT / GM) {
                        T z[GM];
#pragma unroll
                        for (int e = 0; e < GM; ++e) z[e] = tile[g * GM + e][row][wt];
                        *reinterpret_cast<VM*>(outC + (long long)wt * L::CS + L::CO + ((f0 / GM + g) * R + row) * GM) =
                            *reinterpret_cast<VM*>(z);
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// the sweeps
// ---------------------------------------------------------------------------
struct WaveArgs {
    const int4* tasks;          // (plane, first strip, strips, forward index of the plane's strip 0)
    int ntasks;
    const long long* step_off;  // per forward strip: first step block of its records (padding included)
    void* X;
    void* C;
    void* xfer;                 // per task: its published hand-off columns
    long long xstride;          // elements per task
    int* progress;              // per task: hand-off chunks published
    int* ticket;
};

namespace {

__device__ __forceinline__ void give_up(const View& v, int* s_bail) {
    *reinterpret_cast<volatile int*>(s_bail) = 1;
    atomicExch(&v.sc->spin_abort, 1ull);
    atomicMax(&v.sc->status, SCFD_E_SPIN);
}
__device__ __forceinline__ bool aborted(const View& v, const int* s_bail) {
    return *reinterpret_cast<const volatile int*>(s_bail) != 0 ||
           *reinterpret_cast<const volatile unsigned long long*>(&v.sc->spin_abort) != 0ull;
}
// bounded wait on a phase of a local mbarrier.  Every phase these kernels wait
// for completes on the waiting CTA's own barrier (bulk-copy transaction counts,
// or arrivals that carry no data the waiter reads from another CTA), so CTA-scope
// acquire is enough.
__device__ __forceinline__ bool wait_phase(unsigned long long* bar, unsigned par, const View& v, const int* s_bail) {
    // a phase that has already completed is seen by the non-blocking test
    // cheaper than by try_wait (about 50 cycles less per wait in the sweeps)
    if (mbar_test_wait(bar, par)) return true;
    long long spins = 0;
    while (!mbar_try_wait(bar, par)) {
        if (++spins > kSpin || ((spins & 1023) == 0 && aborted(v, s_bail))) return false;
    }
    return true;
}

// a lane's share of one cell's record
template <typename RT, int NY, int PRE>
struct Rec {
    using L = WL<RT, NY, PRE>;
    using CM = typename L::CM;
    RT x[L::K], own[L::NP * L::GP], cm[L::NM * L::GM];
    RT x4[NY == 1 && PRE != 0 ? 4 : 1];  // the cell's four components (dual's S on the backward sweep)
    template <int G>
    static __device__ __forceinline__ void vec(RT* d, const RT* s) {
        using V = typename VecOf<RT, G>::type;
        *reinterpret_cast<V*>(d) = *reinterpret_cast<const V*>(s);
    }
    // the parts that the sweep direction reads
    template <int DIR>
    __device__ __forceinline__ void load(const RT* sx, const RT* sc, int lane, int row) {
        constexpr int GM = L::GM, GP = L::GP;
        const RT* pm = sc + L::CO + row * GM;
        vec<GM>(&cm[0], pm);
#pragma unroll
        for (int k = 0; k < L::K; ++k) x[k] = sx[k * 32 + lane];
        if constexpr (NY == 1 && PRE != 0 && DIR == 1) {
#pragma unroll
            for (int g = 0; g < 4 / GM; ++g) vec<GM>(&x4[g * GM], sx + row * LPC + g * GM);
        }
#pragma unroll
        for (int g = 0; g < L::NP; ++g) vec<GP>(&own[g * GP], sc + (g * 32 + lane) * GP);
#pragma unroll
        for (int g = 1; g < L::NM; ++g) {
            const int f = g * GM;
            const bool both = f < CM::FWD || f >= CM::PRE;
            const bool fwd = f >= CM::FWD && f < CM::BWD, bwd = f >= CM::BWD && f < (PRE ? CM::BWD_END : CM::LMB + 1);
            if (both || (DIR == 0 && fwd) || (DIR == 1 && bwd)) vec<GM>(&cm[f], pm + g * R * GM);
        }
    }
};

__device__ __forceinline__ double mul_add(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mul_add(float a, float b, float c) { return fmaf(a, b, c); }

// sum of a[B..E) as a balanced pairwise tree (short dependency chain)
template <int B, int E, typename RT>
__device__ __forceinline__ RT tree_sum(const RT* a) {
    if constexpr (E - B == 1)
        return a[B];
    else
        return tree_sum<B, (B + E) / 2>(a) + tree_sum<(B + E) / 2, E>(a);
}

// One sweep step of a lane, in two parts.  front(): x of its components from the
// record and the neighbours' products (oA: this lane's of the cell before; sh: the row
// below's of the step before; xv: the strip below's, used by row 0), then its product
// oB, which the next step's shuffles wait for.  back(): its product oA.
//   o = (Y, u, v, H) fb + (fa lam) x + (fa n1, fa n2, fa un) P,
// ds/2 folded into the direction's coefficients (k_pack).
template <typename RT, int NY, int PRE, int DIR, int Q2D>
struct CellStep {
    using L = WL<RT, NY, PRE>;
    using CM = typename L::CM;
    static constexpr unsigned ALL = 0xffffffffu;
    RT x[L::K], xu, xw, S, P;  // P: dpdq.x, S: the species' sum, xu, xw: rho u, rho v

    // the product of direction d (0: A, 1: B) of slot k
    __device__ __forceinline__ void product(const Rec<RT, NY, PRE>& r, int d, RT mE, RT* o) const {
        const RT p1 = r.cm[d == 0 ? CM::P1A : CM::P1B], p2 = r.cm[d == 0 ? CM::P2A : CM::P2B],
                 pu = r.cm[d == 0 ? CM::PUA : CM::PUB];
        const RT fl = r.cm[DIR == 0 ? (d == 0 ? CM::LPA : CM::LPB) : (d == 0 ? CM::LMA : CM::LMB)];
        if constexpr (NY == 1) {
            RT fb = p1 * xu + p2 * xw - pu * S;
            // (I + s2 p1 p2^T) z: p2.z = (p2.p1) fb + pu P, since p2.(0, n1, n2, un) = 0
            if constexpr (PRE != 0) fb = mul_add(r.cm[CM::K1], fb, r.cm[CM::S2] * pu * P);
            o[0] = r.own[0] * fb + fl * x[0] + r.own[1 + d] * P;
        } else {
            // the factors of P of the lanes that hold species are zero
            const RT fb = mul_add(p2, xw, mul_add(p1, xu, -pu * S));
            o[0] = mul_add(r.own[1], fb, mul_add(mE * p1, P, fl * x[0]));
            o[1] = mul_add(r.own[3], fb, mul_add(mE * p2, P, fl * x[1]));
            o[2] = mul_add(r.own[5], fb, mul_add(mE * pu, P, fl * x[2]));
        }
    }

    __device__ __forceinline__ void front(const Rec<RT, NY, PRE>& r, int lane, RT mE, const RT* sh, const RT* xv, const RT* oA,
                                          RT* oB) {
        const int sub = lane % LPC;
        const bool row0 = lane < LPC;
        const RT al = r.cm[CM::AL];
        if constexpr (NY == 1) {
            const RT inB = row0 ? xv[0] : sh[0];
            RT xo, xs[4];
            if constexpr (PRE == 0) {
                xo = DIR == 0 ? al * (r.x[0] + (oA[0] + inB)) : r.x[0] - al * (oA[0] + inB);
            } else {
                RT rv = r.x[0];
                if (DIR == 1) {
                    // dual's S on the forward result (time_dual_viscous.f90:62-68)
                    const RT g = r.cm[CM::S3] * (r.cm[CM::D0] * r.x4[0] + r.cm[CM::DU] * r.x4[1] +
                                                 (r.cm[CM::DV] * r.x4[2] + r.cm[CM::DE] * r.x4[3]));
                    rv = r.cm[CM::S1] * mul_add(g, r.own[0], rv);
                }
                xo = mul_add(DIR == 0 ? al : -al, oA[0] + inB, rv);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) xs[k] = __shfl_sync(ALL, xo, (lane & ~(LPC - 1)) | k);
            if constexpr (PRE != 0) {
                // dual's S^-1 (time_dual_viscous.f90:50-51, 84-85); s4 = 0, 1/s1 = 1 for precon
                const RT g = r.cm[CM::S4] * (r.cm[CM::D0] * xs[0] + r.cm[CM::DU] * xs[1] +
                                             (r.cm[CM::DV] * xs[2] + r.cm[CM::DE] * xs[3]));
                xo = r.cm[CM::I1] * mul_add(g, r.own[0], xo);
#pragma unroll
                for (int k = 0; k < 4; ++k) xs[k] = r.cm[CM::I1] * mul_add(g, r.cm[CM::Y0 + k], xs[k]);
            }
            // P = dpdq.x; forward q2d: the semi-implicit pressure source
            // (time_lusgs_viscous.f90:38-44).  The order of these sums stays as it is: a
            // flow that runs thousands of iterations amplifies rounding.
            const RT pr[3] = {r.cm[CM::D0] * xs[0], r.cm[CM::DU] * xs[1], r.cm[CM::DE] * xs[3]};
            P = tree_sum<0, 3>(pr);
            if (DIR == 0 && Q2D) {
                xs[2] = (xs[2] + r.cm[CM::AA] * P) * r.cm[CM::RQ];
                xo = sub == 2 ? xs[2] : xo;
            }
            P += r.cm[CM::DV] * xs[2];
            x[0] = xo;
            S = xs[0];
            xu = xs[1];
            xw = xs[2];
        } else {
            const RT sal = DIR == 0 ? al : -al;
            const RT alB = row0 ? RT(0) : sal, al0 = row0 ? sal : RT(0);
#pragma unroll
            for (int k = 0; k < 3; ++k) x[k] = mul_add(alB, sh[k], mul_add(al0, xv[k], mul_add(sal, oA[k], r.x[k])));
            const RT* const dp = r.own;  // (dpdq, primitive) pairs; dpdq of rho v is zero
            // without the pressure source its factor joins the lane's sum, otherwise
            // rho v's share follows it
            const RT d1 = Q2D ? dp[2] : mul_add(mE, r.cm[CM::DV], dp[2]);
            P = mul_add(dp[4], x[2], mul_add(d1, x[1], dp[0] * x[0]));
            P += __shfl_xor_sync(ALL, P, 1);
            xw = __shfl_sync(ALL, x[1], lane | 3);
            P += __shfl_xor_sync(ALL, P, 2);
            xu = __shfl_sync(ALL, x[0], lane | 3);
            S = (RT(1) - mE) * ((x[0] + x[1]) + x[2]);
            S += __shfl_xor_sync(ALL, S, 1);
            S += __shfl_xor_sync(ALL, S, 2);
            if (Q2D) {
                // (q2d time_lusgs_viscous.f90:38-44) xw' = (xw + AA P) RQ, P' = P + DV xw'
                const RT rq = r.cm[CM::RQ], aq = r.cm[CM::AA] * rq, dv = r.cm[CM::DV];
                const RT P0 = P, w0 = rq * xw;
                xw = mul_add(aq, P0, w0);
                P = mul_add(mul_add(dv, aq, RT(1)), P0, dv * w0);
                x[1] = sub == 3 ? xw : x[1];
            }
        }
        product(r, 1, mE, oB);
    }
    __device__ __forceinline__ void back(const Rec<RT, NY, PRE>& r, RT mE, RT* oA) const { product(r, 0, mE, oA); }
};

}  // namespace

// one CTA per SM (its shared memory)
template <typename RT, int NY, int PRE, int DIR, int Q2D>
__global__ void __launch_bounds__(kThreads, 1) k_wave(View v, WaveArgs a) {
    using L = WL<RT, NY, PRE>;
    constexpr int XS = L::XS, CSZ = L::CS, D4 = L::D4, K = L::K, PFB = L::PFB;
    constexpr unsigned CHUNK_BYTES = HK * D4 * sizeof(RT);
    static_assert(SPB <= kPadSteps, "a record slot may reach into the padding by at most one slot");
    static_assert((CHUNK_BYTES % 16) == 0 && (SPB * XS * sizeof(RT)) % 16 == 0 && (CSZ * sizeof(RT)) % 16 == 0,
                  "bulk copies are whole 16-byte vectors");
    extern __shared__ __align__(128) unsigned char sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the strip this warp works for (warp 6: the first)
    const int unit = warp != kWarpIn ? warp % UPC : 0;
    struct Unit {
        RT *ringX, *ringC;  // [PFB][SPB][XS], [PFB][SPB][CS]
        RT *xin, *xout;     // [HS][HK][D4]: columns from the strip below; top row for the next strip
        unsigned long long *rfull, *rdone;  // record slot loaded (expect_tx + bulk copies) / read (compute warp)
        unsigned long long* xfull;   // hand-off chunk arrived (bulk copy, or the first strip's top row)
        unsigned long long* pempty;  // a chunk this strip produced is consumed (or published in global memory)
        unsigned long long* hempty;  // a chunk fetched from global memory is consumed
        unsigned long long* oful;    // xout chunk written (the top row's four lanes)
    };
    auto unit_at = [&](int n) {
        Unit q;
        unsigned char* m = sm + n * L::UNIT;
        q.ringX = reinterpret_cast<RT*>(m);
        q.ringC = q.ringX + PFB * SPB * XS;
        q.xin = q.ringC + PFB * SPB * CSZ;
        q.xout = q.xin + HS * HK * D4;
        q.rfull = reinterpret_cast<unsigned long long*>(q.xout + HS * HK * D4);
        q.rdone = q.rfull + PFB;
        q.xfull = q.rdone + PFB;
        q.pempty = q.xfull + HS;
        q.hempty = q.pempty + HS;
        q.oful = q.hempty + HS;
        return q;
    };
    const Unit U = unit_at(unit), Uo = unit_at(unit ^ 1);
    int* s_task = reinterpret_cast<int*>(sm + UPC * L::UNIT);
    int* s_bail = s_task + 1;

    __shared__ __align__(16) RT s_zero[HK * D4];  // the strip-below columns where there are none
    const unsigned rank = cluster_rank();
    if (threadIdx.x < HK * D4) s_zero[threadIdx.x] = RT(0);
    // columns beyond a plane's last chunk are read (times alpha = 0) but never written
    for (int k = threadIdx.x; k < UPC * HS * HK * D4; k += kThreads)
        unit_at(k / (HS * HK * D4)).xin[k % (HS * HK * D4)] = RT(0);
    // every barrier once: a second init of a live mbarrier is undefined
    for (int k = threadIdx.x; k < UPC * L::NBAR; k += kThreads)
        mbar_init(&unit_at(k / L::NBAR).rfull[k % L::NBAR], L::arrivals(k / L::NBAR, k % L::NBAR));
    mbar_init_fence();
    if (threadIdx.x == 0) {
        *s_bail = 0;
        *s_task = 0;
    }
    fence_proxy_async_smem();
    __syncthreads();
    cluster_sync();

    // running uses (over all tasks of this cluster) of this strip's rings
    unsigned rc = 0;  // record slots
    unsigned xc = 0;  // hand-off chunks consumed from xin
    unsigned pc = 0;  // chunks of this strip's top row

    for (;;) {
        if (threadIdx.x == 0 && rank == 0) {
            int t = atomicAdd(a.ticket, 1);
            if (aborted(v, s_bail)) t = a.ntasks;
            *s_task = t;
        }
        cluster_sync();
        int task;
        {
            const unsigned ra = mapa(s_task, 0);
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(task) : "r"(ra) : "memory");
        }
        if (task >= a.ntasks) break;
        const int4 tk = a.tasks[task];
        const int p = tk.x, s0 = tk.y, ns = tk.z, fsb = tk.w;
        const int ni = v.P.ni[p], nstr = (v.P.nj[p] + R - 1) / R;
        const int pos = (int)rank * UPC + unit;  // this strip's place in the task
        const bool active = pos < ns;
        const int strip = DIR == 0 ? s0 + pos : s0 - pos;
        const bool pred_task = DIR == 0 ? s0 > 0 : s0 < nstr - 1;
        const bool succ_task = DIR == 0 ? s0 + ns < nstr : s0 - ns >= 0;
        const bool has_prev = active && (pos > 0 || pred_task);
        const bool pub_next = active && pos + 1 < ns;
        const bool pub_global = active && pos + 1 == ns && succ_task;
        const int nsteps = ni + R - 1;
        const int nch = (nsteps + SPB - 1) / SPB;
        const int nxc = chunks_of(ni);
        const long long sbase = active ? a.step_off[fsb + strip] + kPadSteps : 0;

        if (warp < UPC && active) {
            // ------------------------------------------------------------ a strip's wavefront
            bool bail = false;
            const int row = lane / LPC;
            const int mrow = DIR == 0 ? row : R - 1 - row;  // this lane's row in a step block
            const int mlane = mrow * LPC + lane % LPC;
            // results: this lane's values of step t in X
            RT* gx = reinterpret_cast<RT*>(a.X) + (sbase + (DIR == 0 ? 0 : nsteps - 1)) * XS + mlane;
            const RT mE = lane % LPC == 3 ? RT(1) : RT(0);  // the lane of rho u, rho v, rho E (8, 9 species)
            RT outA[K], outB[K], sh[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                outA[k] = RT(0);
                sh[k] = RT(0);
            }
            // The hand-off.  Chunk j of the strip below holds the columns 4j-3 .. 4j
            // (HK = 4) of its top row: its row R-1 computes column c at its step c + R-1,
            // so its group of steps g (4g .. 4g+3) yields exactly chunk g - (R/4 - 1).  Row 0
            // here uses column t at step t: chunk g's last column at step 4g (u = 0 of
            // group g), chunk g+1's first three at u = 1..3, so chunk g+1 is awaited
            // between u = 0 and u = 1.
            static_assert(HK == 4 && SPB % HK == 0 && R % HK == 0, "groups of 4 steps, whole groups per record slot");
            const int lastc = nxc - 1;
            auto chunk_test = [&](unsigned k) { return mbar_test_wait(&U.xfull[k % HS], (k / HS) & 1u); };
            auto await_chunk = [&](unsigned k) -> bool {
                return __all_sync(0xffffffffu, wait_phase(&U.xfull[k % HS], (k / HS) & 1u, v, s_bail));
            };
            auto await_slot = [&](unsigned n) -> bool {
                return __all_sync(0xffffffffu, wait_phase(&U.rfull[n % PFB], (n / PFB) & 1u, v, s_bail));
            };
            if ((has_prev && !await_chunk(xc)) || !await_slot(rc)) bail = true;
            // the record of the step at hand and of the next one
            Rec<RT, NY, PRE> rec[2];
            if (!bail) {
                const unsigned o = (rc % PFB) * SPB + (DIR == 0 ? 0 : SPB - 1);
                rec[0].template load<DIR>(U.ringX + o * XS, U.ringC + o * CSZ, mlane, mrow);
            }
            const bool pub_any = pub_next || pub_global;
            // the top row goes straight into the next strip's ring where that is this CTA's, else
            // to the warp that passes it on
            const bool direct = pub_next && unit == 0;
            RT* const oring = direct ? Uo.xin : U.xout;
            unsigned long long* const obar = direct ? Uo.xfull : U.oful;
            unsigned pfree = pc + 1;  // chunks before this one may be written
            // A wait splits the code that the compiler can schedule (120-180 cycles per
            // wait in a loop of 4 steps), so a slot of 8 steps has three: for the chunk of each
            // group, tested a step ahead, and for the next slot; stores and arrivals of some
            // lanes are predicated, without branches.
            for (int n = 0; n < nch && !bail; ++n) {
                const unsigned slot = rc % PFB;
                const RT* sx = U.ringX + slot * SPB * XS;
                const RT* sc = U.ringC + slot * SPB * CSZ;
                // back-pressure: chunk k reuses the place of chunk k - HS, and chunks are
                // released in order, so the release of chunk pc + 7 - HS covers this slot's two
                // and the next six
                if (pub_any && pc + 1 >= pfree) {
                    const unsigned pw = pc + 7u;
                    if (pw >= HS && !__all_sync(0xffffffffu, wait_phase(&U.pempty[pw % HS], ((pw / HS) - 1u) & 1u, v, s_bail))) {
                        bail = true;
                        break;
                    }
                    pfree = pw + 1;
                }
#pragma unroll
                for (int h = 0; h < SPB / HK; ++h) {
                    const int g = n * (SPB / HK) + h;
                    // this group's top-row outputs form chunk J of the strip above
                    const int J = g - (R / 4 - 1);
                    const bool pub = pub_any && J >= 0 && J <= lastc;
                    const bool put = pub && row == R - 1;
                    const unsigned ps = pc % HS;
                    // the strip below's columns: chunk g's last, then chunk g+1's first three (a
                    // zero column where there is no strip)
                    const RT* const cA = has_prev ? U.xin + ((xc + g) % HS * HK + 3) * D4 + lane % LPC * K : s_zero;
                    const RT* const cB = has_prev ? U.xin + (xc + g + 1) % HS * HK * D4 + lane % LPC * K : s_zero;
                    RT* const xo = oring + ps * HK * D4 + lane % LPC * K;
#pragma unroll
                    for (int u = 0; u < HK; ++u) {
                        const int s = h * HK + u;  // step of the slot
                        Rec<RT, NY, PRE>& cur = rec[s & 1];
                        Rec<RT, NY, PRE>& nxt = rec[(s + 1) & 1];
                        const RT* xi = u == 0 ? cA : cB + (u - 1) * D4;
                        RT xv[K];
#pragma unroll
                        for (int k = 0; k < K; ++k) xv[k] = xi[k];
                        bool ready = true;
                        if (u == 0 && has_prev && g + 1 <= lastc) ready = chunk_test(xc + g + 1);
                        if (s + 1 == SPB && n + 1 < nch)
                            ready = mbar_test_wait(&U.rfull[(rc + 1) % PFB], ((rc + 1) / PFB) & 1u);
                        CellStep<RT, NY, PRE, DIR, Q2D> st;
                        st.front(cur, lane, mE, sh, xv, outA, outB);
                        // for the next step: the row below's products, the record (the last step of
                        // a slot has all its records in registers: the slot is free)
#pragma unroll
                        for (int k = 0; k < K; ++k) sh[k] = __shfl_up_sync(0xffffffffu, outB[k], LPC);
                        if (s + 1 < SPB) {
                            const int q = DIR == 0 ? s + 1 : SPB - 2 - s;
                            nxt.template load<DIR>(sx + q * XS, sc + q * CSZ, mlane, mrow);
                        } else {
                            __syncwarp();
                            mbar_arrive_if(&U.rdone[slot], lane == 0);
                            ++rc;
                            if (!__all_sync(0xffffffffu, ready) && !await_slot(rc)) {
                                bail = true;
                                break;
                            }
                            const unsigned o = (rc % PFB) * SPB + (DIR == 0 ? 0 : SPB - 1);
                            if (n + 1 < nch) nxt.template load<DIR>(U.ringX + o * XS, U.ringC + o * CSZ, mlane, mrow);
                        }
                        st.back(cur, mE, outA);
                        // steps past the last one fall into the padding
#pragma unroll
                        for (int k = 0; k < K; ++k) gx[(DIR == 0 ? s : -s) * XS + k * 32] = st.x[k];
                        // the top row: entry u of chunk J in this strip's xout ring
#pragma unroll
                        for (int k = 0; k < K; ++k) st_shared_if(xo + u * D4 + k, outB[k], put);
                        if (u == 0 && !__all_sync(0xffffffffu, ready) && !await_chunk(xc + g + 1)) {
                            bail = true;
                            break;
                        }
                    }
                    if (bail) break;
                    // chunk J complete: on to the warp that passes it on.
                    // Columns outside 0 .. ni-1 travel as they are.
                    mbar_arrive_if(&obar[ps], put);
                    pc += pub ? 1u : 0u;
                }
                gx += (DIR == 0 ? SPB : -SPB) * XS;
            }
            if (has_prev) xc += nxc;
            if (bail && lane == 0) give_up(v, s_bail);
        } else if (warp >= kWarpLoad && warp < kWarpLoad + UPC && active) {
            // ------------------------------------------------------------ record loads, chunk releases
            if (lane == 0) {
                const RT* gX = reinterpret_cast<const RT*>(a.X) + sbase * XS;
                const RT* gC = reinterpret_cast<const RT*>(a.C) + sbase * CSZ;
                // consumed chunks are released to the strip below (its pempty) or to the warp
                // that fetched them
                const unsigned rel = pos == 0 ? mapa(U.hempty, rank)
                                              : mapa(Uo.pempty, unit == 0 ? rank - 1 : rank);
                auto slot_done = [&](int m) -> bool {
                    const unsigned k = rc + m;
                    if (!wait_phase(&U.rdone[k % PFB], (k / PFB) & 1u, v, s_bail)) return false;
                    // slot m's steps read the columns up to 8 m + 7: chunks 2 m, 2 m + 1 are used up.
                    // A chunk is refilled HS chunks later, long after these reads.
                    if (has_prev)
                        for (int q = 2 * m; q < 2 * m + 2 && q < nxc; ++q)
                            mbar_arrive_cluster_relaxed(rel + ((xc + q) % HS) * 8u);
                    return true;
                };
                static_assert(SPB == 2 * HK, "two chunks per slot");
                int nl = 0;
                bool ok = true;
                for (; nl < nch; ++nl) {
                    const unsigned k = rc + nl, slot = k % PFB;
                    // the slot is free once its last records are in registers
                    if (nl >= PFB && !(ok = slot_done(nl - PFB))) break;
                    const long long st0 = DIR == 0 ? (long long)nl * SPB : (long long)(nsteps - 1) - (long long)nl * SPB - (SPB - 1);
                    mbar_expect_tx(&U.rfull[slot], SPB * (XS + CSZ) * sizeof(RT));
                    tma_bulk_g2s(U.ringX + slot * SPB * XS, gX + st0 * XS, SPB * XS * sizeof(RT), &U.rfull[slot]);
                    tma_bulk_g2s(U.ringC + slot * SPB * CSZ, gC + st0 * CSZ, SPB * CSZ * sizeof(RT), &U.rfull[slot]);
                }
                // every load has landed and every slot is free before the next task (or the
                // CTA's end)
                for (int m = nl > PFB ? nl - PFB : 0; m < nl; ++m) {
                    const unsigned k = rc + m;
                    long long spins = 0;
                    while (!mbar_try_wait(&U.rfull[k % PFB], (k / PFB) & 1u) && ++spins < kSpin) {
                    }
                    if (ok) ok = slot_done(m);
                }
                if (!ok) give_up(v, s_bail);
            }
            __syncwarp();
            rc += nch;
            if (has_prev) xc += nxc;
        } else if (warp >= kWarpOut && warp < kWarpOut + UPC && pub_next) {
            // ------------------------------------------------------------ hand-off to the next strip
            // one bulk copy per chunk into its ring, completing the receiver's barrier
            // phase with this arrival and the copy's bytes (in either order)
            if (lane == 0 && unit == UPC - 1) {
                const unsigned dring = mapa(Uo.xin, rank + 1), dfull = mapa(Uo.xfull, rank + 1);
                for (int h = 0; h < nxc; ++h) {
                    const unsigned k = pc + h, ps = k % HS;
                    if (!wait_phase(&U.oful[ps], (k / HS) & 1u, v, s_bail)) {
                        give_up(v, s_bail);
                        break;
                    }
                    fence_proxy_async_smem();
                    mbar_arrive_expect_tx_cluster_relaxed(dfull + ps * 8u, CHUNK_BYTES);
                    bulk_s2dsmem(dring + ps * CHUNK_BYTES, U.xout + ps * HK * D4, CHUNK_BYTES, dfull + ps * 8u);
                }
            }
            __syncwarp();
            pc += nxc;
        } else if (warp >= kWarpOut && warp < kWarpOut + UPC && pub_global) {
            // ------------------------------------------------------------ hand-off out, through global memory
            RT* xdst = reinterpret_cast<RT*>(a.xfer) + (long long)task * a.xstride;
            int* prog_out = a.progress + task;
            int h = 0;
            while (h < nxc) {
                const unsigned k = pc + h;
                bool ok = wait_phase(&U.oful[k % HS], (k / HS) & 1u, v, s_bail);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) give_up(v, s_bail);
                    break;
                }
                // this chunk and those after it that are ready too, under one fence
                int m = 1;
                while (m < 8 && h + m < nxc) {
                    ok = mbar_test_wait(&U.oful[(k + m) % HS], ((k + m) / HS) & 1u);
                    if (!__all_sync(0xffffffffu, ok)) break;
                    ++m;
                }
                for (int q = 0; q < m; ++q)
                    for (int e = lane; e < HK * D4; e += 32)
                        xdst[(long long)(h + q) * HK * D4 + e] = U.xout[((k + q) % HS) * HK * D4 + e];
                __threadfence();
                __syncwarp();
                if (lane == 0) {
                    st_release_gpu(prog_out, h + m);
                    for (int q = 0; q < m; ++q) mbar_arrive(&U.pempty[(k + q) % HS]);
                }
                __syncwarp();
                h += m;
            }
            pc += nxc;
        } else if (warp == kWarpIn && active && pos == 0 && pred_task) {
            // ------------------------------------------------------------ hand-off in, through global memory
            if (lane == 0) {
                const int* prog_in = a.progress + (task - 1);
                const RT* xsrc = reinterpret_cast<const RT*>(a.xfer) + (long long)(task - 1) * a.xstride;
                int seen = 0, h = 0;
                bool ok = true;
                for (; h < nxc; ++h) {
                    if (seen <= h) {
                        long long spins = 0;
                        while ((seen = ld_acquire_gpu(prog_in)) <= h) {
                            if (++spins > kSpin || ((spins & 255) == 0 && aborted(v, s_bail))) {
                                ok = false;
                                break;
                            }
                        }
                        fence_proxy_async_global();
                    }
                    const unsigned k = xc + h, hs = k % HS;
                    if (ok && k >= HS) ok = wait_phase(&U.hempty[hs], ((k / HS) - 1u) & 1u, v, s_bail);
                    if (!ok) {
                        give_up(v, s_bail);
                        break;
                    }
                    mbar_expect_tx(&U.xfull[hs], CHUNK_BYTES);
                    tma_bulk_g2s(U.xin + hs * HK * D4, xsrc + (long long)h * HK * D4, CHUNK_BYTES, &U.xfull[hs]);
                }
                // chunks in flight land before the CTA's end (the last HS at most)
                for (int m = h > HS ? h - HS : 0; m < h; ++m) {
                    const unsigned k = xc + m;
                    long long spins = 0;
                    while (!mbar_try_wait(&U.xfull[k % HS], (k / HS) & 1u) && ++spins < kSpin) {
                    }
                }
            }
            __syncwarp();
            xc += nxc;
        }
        cluster_sync();  // the task is done in every CTA of the cluster
    }
    // Where every wait came true, every chunk copied into this CTA's rings has been waited for.
    // After one that gave up, chunks may still be on their way: their copies end (within a
    // microsecond) before any CTA of the cluster leaves.
    if (*reinterpret_cast<volatile int*>(s_bail) != 0)
        for (const long long t0 = clock64(); clock64() - t0 < kDrain;) {
        }
    cluster_sync();  // no CTA leaves while a peer may still reach its shared memory
}

// ---------------------------------------------------------------------------
// Records -> cells, for a block of 32 steps x R rows of one strip: a warp reads
// whole step blocks (all of them before the barrier), then every thread has the
// components of its cell (step x, row y), along i.
// ---------------------------------------------------------------------------
template <typename T, int NY, int PRE>
__device__ __forceinline__ void records_to_tile(const T* in, int nt, T (*tile)[R][33]) {
    using L = WL<T, NY, PRE>;
    constexpr int K = L::K;
    const int ln = threadIdx.x, row = ln / LPC, sub = ln % LPC;
    T z[4][K];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int wt = threadIdx.y + r * R;
#pragma unroll
        for (int k = 0; k < K; ++k) z[r][k] = wt < nt ? in[(long long)wt * L::XS + k * 32 + ln] : T(0);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int m = L::comp(sub, k);
            if (m >= 0) tile[m][row][threadIdx.y + r * R] = z[r][k];
        }
}

// k_omega: the NR relaxation's candidates from the backward sweep's result
// (time_NR_viscous.f90:56-78): per block of 32 steps x R rows of a strip,
// res = sum of Dq(E)^2 and omega = min over Dq_k < 0 of -q_k / Dq_k * Dqmax,
// into partials[2 b], partials[2 b + 1]; the block that finishes last reduces them
// in fixed order into the pair after the last block's (every block of k_unpack
// reading all 3264 pairs of the 786 k-cell step would move 170 MB).
template <typename T, int NY, int PRE>
__global__ void __launch_bounds__(32 * R)
k_omega(View v, const int2* blk, const int4* strips, const long long* step_off, const T* X, double* partials,
        int* counter) {
    using L = WL<T, NY, PRE>;
    __shared__ T tile[L::D][R][33];
    __shared__ double sred[2][R];
    __shared__ bool s_last;
    const int2 b = blk[blockIdx.x];
    const int4 st = strips[b.x];
    const int p = st.x, s = st.y;
    const int ni = v.P.ni[p], nj = v.P.nj[p];
    const int nt = min(32, ni + R - 1 - b.y);
    const long long N = v.ncell;
    const int tt = threadIdx.x, l = threadIdx.y;
    const int t = b.y + tt, cc = t - l, j = R * s + 1 + l;
    const bool wr = tt < nt && cc >= 0 && cc < ni && j <= nj;
    const long long c = wr ? cidx(v.P, p, cc + 1, j) : 0;
    double qr[NY];
#pragma unroll
    for (int m = 0; m < NY; ++m) qr[m] = wr ? v.q[m * N + c] : 0.0;
    records_to_tile<T, NY, PRE>(X + (step_off[b.x] + kPadSteps + b.y) * L::XS, nt, tile);
    __syncthreads();
    double res = 0.0, om = 1e300;
    if (wr) {
#pragma unroll
        for (int m = 0; m < NY; ++m) {
            const double dq = double(tile[m][l][tt]);
            if (dq < 0.0) om = fmin(om, -qr[m] / dq * v.dq_max);
        }
        const double dE = double(tile[NY + 2][l][tt]);
        res = dE * dE;
    }
    double* out = partials + 2 * blockIdx.x;
    // the block's cells in a fixed order: warps, then lanes
    for (int d = 16; d > 0; d >>= 1) {
        res += __shfl_down_sync(0xffffffffu, res, d);
        om = fmin(om, __shfl_down_sync(0xffffffffu, om, d));
    }
    if (threadIdx.x == 0) {
        sred[0][threadIdx.y] = res;
        sred[1][threadIdx.y] = om;
    }
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        for (int k = 1; k < R; ++k) {
            res += sred[0][k];
            om = fmin(om, sred[1][k]);
        }
        out[0] = res;
        out[1] = om;
        __threadfence();
        s_last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        reduce_partials(partials, gridDim.x, res, om);
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            partials[2 * gridDim.x] = res;
            partials[2 * gridDim.x + 1] = om;
        }
    }
}

// ---------------------------------------------------------------------------
// k_unpack: q += omega * Dq from the records (LU-SGS: omega = 1; NR: the
// positivity-limited omega of k_omega, time_NR_viscous.f90:86-108).
// ---------------------------------------------------------------------------
template <typename T, int NY, int PRE>
__global__ void __launch_bounds__(32 * R)
k_unpack(View v, const int2* blk, const int4* strips, const long long* step_off, const T* X, const double* partials,
         int nr_mode, int inner) {
    using L = WL<T, NY, PRE>;
    constexpr int D = L::D;
    __shared__ T tile[D][R][33];
    const int2 b = blk[blockIdx.x];
    const int4 st = strips[b.x];
    const int p = st.x, s = st.y;
    const int ni = v.P.ni[p], nj = v.P.nj[p];
    const int nt = min(32, ni + R - 1 - b.y);
    const long long N = v.ncell;
    const int tt = threadIdx.x, l = threadIdx.y;
    const int t = b.y + tt, cc = t - l, j = R * s + 1 + l;
    const bool wr = tt < nt && cc >= 0 && cc < ni && j <= nj;
    const long long c = wr ? cidx(v.P, p, cc + 1, j) : 0;
    // every record value and q of the block's cells are loaded before the first
    // barrier, so that the loads overlap one another
    double qr[D];
#pragma unroll
    for (int k = 0; k < D; ++k) qr[k] = wr ? v.q[k * N + c] : 0.0;
    records_to_tile<T, NY, PRE>(X + (step_off[b.x] + kPadSteps + b.y) * L::XS, nt, tile);
    __syncthreads();
    double om = 1.0;
    if (nr_mode) {
        // (res, omega) of all blocks, or of all ranks
        const double res = partials[0], o = partials[1];
        if (blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
            if (o < v.omega_min) atomicMax(&v.sc->status, SCFD_E_OMEGA);
            if (inner == 1) v.sc->res1 = res;
            v.sc->res = res;
            v.sc->omega = fmin(v.omega_max, o);
            log_inner(v.sc, inner, o, res);
        }
        // time_NR_viscous.f90:75-78: below omega_min the step stops without the update
        if (o < v.omega_min || v.sc->status == SCFD_E_OMEGA) return;
        om = fmin(v.omega_max, o);
    }
    if (wr) {
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const double dq = double(tile[k][l][tt]);
            v.q[k * N + c] = nr_mode ? qr[k] + om * dq : qr[k] + dq;
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
int wave_pad_steps() { return kPadSteps; }
int wave_strips_per_task(int cl) { return cl * UPC; }
int wave_handoff_chunk() { return HK; }
int wave_chunks(int ni) { return chunks_of(ni); }
int wave_rows() { return R; }

namespace {
template <typename RT, int NY, int PRE>
WaveSizes sizes_t() {
    using L = WL<RT, NY, PRE>;
    return WaveSizes{L::XS, L::CS, L::D4, L::SMEM};
}
}  // namespace

// The species counts with a sweep here; the preconditioned schemes (pre) have one
// for a single species (they are non-reacting, and an ideal gas has one).
WaveSizes wave_sizes(int ny, bool mixed, bool pre) {
    if (pre) return ny != 1 ? WaveSizes{0, 0, 0, 0} : mixed ? sizes_t<float, 1, 1>() : sizes_t<double, 1, 1>();
    switch (ny) {
        case 1: return mixed ? sizes_t<float, 1, 0>() : sizes_t<double, 1, 0>();
        case 8: return mixed ? sizes_t<float, 8, 0>() : sizes_t<double, 8, 0>();
        case 9: return mixed ? sizes_t<float, 9, 0>() : sizes_t<double, 9, 0>();
        default: return WaveSizes{0, 0, 0, 0};
    }
}

namespace {

cudaLaunchAttribute cluster_of(int cl) {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = cl;
    a.val.clusterDim.y = 1;
    a.val.clusterDim.z = 1;
    return a;
}

// The kernel's attributes are set for every context: they go with the device's primary
// context, which cudaDeviceReset ends.  The count of co-resident clusters is the device's
// own, and its query takes milliseconds, so a process asks once per kernel, device and
// cluster size.
template <typename RT, int NY, int PRE, int DIR, int Q2D>
int max_clusters_t(int cl) {
    using L = WL<RT, NY, PRE>;
    static std::mutex m;
    static std::map<std::pair<int, int>, int> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    const auto kernel = k_wave<RT, NY, PRE, DIR, Q2D>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    std::lock_guard<std::mutex> lock(m);
    const auto it = known.find({dev, cl});
    if (it != known.end()) return it->second;
    cudaLaunchAttribute attr = cluster_of(cl);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cl, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = L::SMEM;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (n > 0) known[{dev, cl}] = n;
    return n;
}

// of the two kernels that a context launches (each is loaded by its query): the forward
// sweep of its dimension and the backward sweep
template <typename RT, int NY, int PRE>
int max_clusters_ny(bool q2d, int cl) {
    int n = max_clusters_t<RT, NY, PRE, 1, 0>(cl);
    if constexpr (PRE == 0) {  // the preconditioned schemes are 2d
        if (q2d) return std::min(n, max_clusters_t<RT, NY, PRE, 0, 1>(cl));
    }
    return std::min(n, max_clusters_t<RT, NY, PRE, 0, 0>(cl));
}

}  // namespace

int wave_max_clusters(int ny, bool mixed, bool pre, bool q2d, int cl) {
    if (pre) return ny != 1 ? 0 : mixed ? max_clusters_ny<float, 1, 1>(q2d, cl) : max_clusters_ny<double, 1, 1>(q2d, cl);
    switch (ny) {
        case 1: return mixed ? max_clusters_ny<float, 1, 0>(q2d, cl) : max_clusters_ny<double, 1, 0>(q2d, cl);
        case 8: return mixed ? max_clusters_ny<float, 8, 0>(q2d, cl) : max_clusters_ny<double, 8, 0>(q2d, cl);
        case 9: return mixed ? max_clusters_ny<float, 9, 0>(q2d, cl) : max_clusters_ny<double, 9, 0>(q2d, cl);
        default: return 0;
    }
}

namespace {

template <typename RT, int NY, int PRE, int DIR, int Q2D>
void sweep_launch(const View& v, cudaStream_t s, const Wave& w) {
    using L = WL<RT, NY, PRE>;
    WaveArgs a{DIR == 0 ? w.tasks_f : w.tasks_b, w.ntasks,    w.step_off, w.X, w.C, w.xfer, w.xstride,
               w.progress + (DIR == 0 ? 0 : w.ntasks), w.tickets + (DIR == 0 ? 0 : 1)};
    const int ncl = w.nclusters < w.ntasks ? w.nclusters : w.ntasks;
    cudaLaunchAttribute attr = cluster_of(w.cluster);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ncl * w.cluster, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = L::SMEM;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_wave<RT, NY, PRE, DIR, Q2D>, v, a);
}

template <typename RT, int NY, int PRE>
void run_t(const View& v, cudaStream_t s, const Wave& w, int what, int inner) {
    const int nr = dual_time_scheme(v.scheme) ? 1 : 0;
    const dim3 block(32, R);
    RT* X = reinterpret_cast<RT*>(w.X);
    switch (what) {
        case 0:
            k_pack<RT, NY, PRE><<<w.nblk, block, 0, s>>>(v, w.blk, w.strips, w.step_off, X, reinterpret_cast<RT*>(w.C), nr,
                                                         w.progress, 2 * w.ntasks, w.tickets);
            break;
        case 1:
            if constexpr (PRE == 0) {
                if (v.dim == SCFD_DIM_Q2D) {
                    sweep_launch<RT, NY, PRE, 0, 1>(v, s, w);
                    break;
                }
            }
            sweep_launch<RT, NY, PRE, 0, 0>(v, s, w);
            break;
        case 2: sweep_launch<RT, NY, PRE, 1, 0>(v, s, w); break;
        case 3:
            k_unpack<RT, NY, PRE><<<w.nblk, block, 0, s>>>(v, w.blk, w.strips, w.step_off, X, w.partials, nr, inner);
            break;
        default:
            k_omega<RT, NY, PRE><<<w.nblk, block, 0, s>>>(v, w.blk, w.strips, w.step_off, X, w.partials, w.tickets + 2);
            break;
    }
}

}  // namespace

// what: 0 pack, 1 forward sweep, 2 backward sweep, 3 unpack/update, 4 the NR
// partials (res, omega) of the backward sweep's result
int launch_wave(const View& v, cudaStream_t s, const Wave& w, int what, int inner) {
    const bool mixed = v.precision == SCFD_PREC_MIXED;
    if (preconditioned_scheme(v.scheme)) {
        if (v.nY != 1) return 0;
        if (mixed) run_t<float, 1, 1>(v, s, w, what, inner); else run_t<double, 1, 1>(v, s, w, what, inner);
        return 1;
    }
    switch (v.nY) {
        case 1: if (mixed) run_t<float, 1, 0>(v, s, w, what, inner); else run_t<double, 1, 0>(v, s, w, what, inner); return 1;
        case 8: if (mixed) run_t<float, 8, 0>(v, s, w, what, inner); else run_t<double, 8, 0>(v, s, w, what, inner); return 1;
        case 9: if (mixed) run_t<float, 9, 0>(v, s, w, what, inner); else run_t<double, 9, 0>(v, s, w, what, inner); return 1;
        default: return 0;
    }
}

}  // namespace scfd
