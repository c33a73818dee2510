// 1D wave-propagation path: the whole claw1 time loop in ONE persistent CTA.
//
// Reference: src/1d/step1.f90:4-170 (in-place Godunov update, limiter,
// correction flux f), src/1d/bc1.f, src/1d/claw1.f:450-583 (time loop; the
// next dt is chosen before the Courant check, unlike claw2).
//
// 1D grids in this code family are small (hundreds to ~2000 cells), so the
// B200 shape is one CTA that keeps q in shared memory (two copies: a step
// reads one and writes the other, so a rejected step is one not switched to).
// One launch replaces ~10^3 step launches and host round trips.
//
// What bounds a step is the latency of its dependent chain, so the chain is
// kept short and split in two.  A warp holds 32 neighbouring cells, two of
// them halo on each side, and writes 28: waves, limiter ratios, correction
// fluxes and fluctuations stay in registers and cross lanes by shuffle.  Waves
// and limited waves do not need dt, so while a warp of its own folds the last
// step's Courant maxima and runs claw1's dt controller (two divisions), the
// others solve the next step's Riemann problems on the new q; a rejected step
// solves the old q's again.  Two barriers per step.
#pragma once
#include "common.cuh"

namespace clawb200 {

constexpr int STRIP1 = 28;  // cells a warp writes

// Threads of the CTA at most: 512 leave a thread 128 registers; a two-wave
// system fits the 64 that 1024 threads leave, which grids of more than 16
// strips take.
template <class S>
__host__ __device__ constexpr int step1_threads() {
    return S::mwaves >= 3 ? 512 : 1024;
}

template <class S>
struct Step1Args {
    typename S::real* q[2];
    const typename S::real* aux;  // [maux][mx+4]
    long long fstride, afstride;
    int mx;
    int bc[2];
    int mthlim[8];
    int order, fwave, capa;
    double dx;
    // source term (src/1d/claw1.f:486-509): src_split 0 none, 1 Godunov, 2
    // Strang; the radial term of examples/acoustics_2d_radial/1drad/src1.f
    int src_split;
    double src_nd1, src_bulk, xlower;  // ndim - 1, bulk, xlower
    ClawCtl* ctl;
    S solver;
};

// q's two copies and aux in shared memory
template <class S>
long long step1_smem_bytes(int mx) {
    return ((long long)2 * S::meqn * mx + (long long)S::maux * (mx + 4)) * (long long)sizeof(typename S::real);
}

// Largest of the warp's values, each >= 0: their bit patterns order as they do.
__device__ __forceinline__ double warp_max_nonneg(double c) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(c);
    const unsigned hi = (unsigned)(b >> 32);
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
    return __longlong_as_double((long long)(((unsigned long long)mh << 32) | ml));
}

// Methods compiled in: one limiter on every wave at order 2 without capacity,
// f-waves or source (taken branches cost a lone warp 30-100 cycles each), and
// one that reads everything at run time.  us a step, run time -> compiled in:
//               minmod         superbee       van Leer       MC
// acoustics 100   1.32 -> 0.92   1.35 -> 0.93   1.41 -> 1.09   1.35 -> 0.92
//           800   2.32 -> 1.84   2.41 -> 1.92   2.48 -> 2.07   2.40 -> 1.91
//          2500   6.17 -> 4.70   6.43 -> 4.88   6.54 -> 5.28   6.37 -> 4.86
// varying   800   2.74 -> 2.19   2.90 -> 2.32   2.92 -> 2.32   2.90 -> 2.32
// advection 800   1.42 -> 1.18   1.46 -> 1.19   1.53 -> 1.26   1.45 -> 1.19
// Euler     800   6.53 -> 5.47   6.71 -> 5.65   6.98 -> 5.89   6.80 -> 5.64
// and 12 to 30 % for each of them at 100 and 2500 cells.
template <int LIM>
struct Method1 {
    static constexpr int lim = LIM;
};
struct Method1Any {
    static constexpr int lim = -1;
};

// SMQ: q and aux in shared memory; else (grids too large for it) the two
// copies are the handle's own buffers in global memory, L2-resident, whose
// accesses __syncthreads orders within the CTA just the same.  The last warp
// is the controller's.
template <class S, class M, bool SMQ, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) step1_kernel(const __grid_constant__ Step1Args<S> A) {
    using real = typename S::real;
    constexpr int ME = S::meqn, MW = S::mwaves, MA = S::maux;
    constexpr int MAX = MA > 0 ? MA : 1;
    constexpr bool ANY = M::lim < 0;
    constexpr unsigned FULL = 0xffffffffu;
    ClawCtl* ctl = A.ctl;
    const int mx = A.mx, n = mx + 4;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[32];
    __shared__ double sh_dt, sh_dtdx;
    __shared__ int sh_act;
    enum { STEP = 0, RETRY = 1, STOP_NEW = 2, STOP_OLD = 3 };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (blockDim.x >> 5) - 1;
    const int nstrips = (mx + STRIP1 - 1) / STRIP1;
    const int cur = ctl->cur;
    real* sq = reinterpret_cast<real*>(smem_raw);  // [2][ME][mx]
    real* sa = sq + 2 * ME * mx;                   // [MA][n]
    const long long fs = SMQ ? mx : A.fstride, afs = SMQ ? n : A.afstride;
    if constexpr (SMQ) {
        const real* qin = A.q[cur];
        for (int i = tid; i < ME * mx; i += blockDim.x) sq[i] = qin[(i / mx) * A.fstride + i % mx];
        for (int i = tid; i < MA * n; i += blockDim.x) sa[i] = A.aux[(i / n) * A.afstride + i % n];
    }
    // a single step (claw_step) is step1 alone: accepted whatever its Courant
    // number, without the source steps that claw1 wraps around it
    const bool single = ctl->mode == CTL_SINGLE;
    const int src_split = ANY && !single ? A.src_split : 0;
    const double dxd = A.dx;
    int buf = SMQ ? 0 : cur;  // q's copy the step reads
    __syncthreads();

    if (warp == nwarps) {  // ------------------------------- controller
        const bool dt_variable = ctl->dt_variable != 0;
        const double tstart = ctl->tstart, tend = ctl->tend, dt_max = ctl->dt_max, cfl_max = ctl->cfl_max,
                     cfl_desired = ctl->cfl_desired;
        const int maxn = ctl->maxn;
        double t = ctl->t, dt = ctl->dt, dtmin = ctl->dtmin, dtmaxs = ctl->dtmax, cfl = 0.0, cflmax = 0.0;
        double told = t;
        int nacc = 0, nrej = 0, act = STEP;
        bool fresh = true;  // a new step, not a retry
        for (;;) {
            if (act < STOP_NEW) {
                if (fresh) {
                    told = t;
                    if (told + dt > tend && tstart < tend) dt = tend - told;
                }
                t = told + dt;
                if (lane == 0) {
                    sh_dt = dt;
                    sh_dtdx = dt / dxd;
                }
            }
            if (lane == 0) sh_act = act;
            __syncthreads();
            if (act >= STOP_NEW) break;
            __syncthreads();
            cfl = warp_max_nonneg(lane < nwarps ? red[lane] : 0.0);
            // claw1: choose the next dt first (src/1d/claw1.f:520-529) ...
            if (dt_variable) {
                if (cfl > 0.0) {
                    dt = fmin(dt_max, dt * cfl_desired / cfl);
                    dtmin = fmin(dt, dtmin);
                    dtmaxs = fmax(dt, dtmaxs);
                } else {
                    dt = dt_max;
                }
            }
            // ... then check the Courant number (src/1d/claw1.f:533-554)
            if (single || cfl <= cfl_max) {
                cflmax = fmax(cfl, cflmax);
                ++nacc;
                fresh = true;
                act = t >= tend || nacc >= maxn ? STOP_NEW : STEP;
            } else {
                t = told;
                fresh = false;
                if (dt_variable) {
                    ++nrej;
                    act = RETRY;
                } else {
                    cflmax = fmax(cfl, cflmax);
                    act = STOP_OLD;
                }
            }
        }
        if (lane == 0) {
            ctl->t = t;
            ctl->dt = dt;
            ctl->cflmax_seen = cflmax;
            ctl->cfl_last = cfl;
            ctl->dtmin = dtmin;
            ctl->dtmax = dtmaxs;
            ctl->n = nacc;
            ctl->nrej = nrej;
            ctl->cur = SMQ ? cur ^ 1 : (cur ^ (nacc & 1));
            ctl->done = 1;
        }
        buf = (SMQ ? 0 : cur) ^ (nacc & 1);
    } else {  // ----------------------------------------------- cells
        const bool order2 = ANY ? A.order != 1 : true;
        const bool many = nstrips > nwarps;  // several strips per warp
        // the source before a Strang step needs dt
        const bool late = many || src_split == 2;
        // this lane's cell of a strip, its source cell under bc1 (src/1d/bc1.f;
        // a wall negates q(2)); once, unless warps take several strips
        int x0 = 0, x = 0, sx = 0;
        bool neg = false;
        real a[MAX], aL[MAX];
        auto cells = [&](int strip) {
            x0 = strip * STRIP1 + lane - 2;
            x = min(x0, mx + 1);
            sx = x;
            neg = false;
            if (x < 0) {
                neg = A.bc[0] == BC_WALL;
                sx = A.bc[0] == BC_PERIODIC ? mx + x : (neg ? -1 - x : 0);
            } else if (x >= mx) {
                neg = A.bc[1] == BC_WALL;
                sx = A.bc[1] == BC_PERIODIC ? x - mx : (neg ? 2 * mx - 1 - x : mx - 1);
            }
#pragma unroll
            for (int k = 0; k < MA; ++k) {
                a[k] = SMQ ? sa[k * n + x + 2] : A.aux[k * afs + x + 2];
                aL[k] = __shfl_up_sync(FULL, a[k], 1);
            }
        };
        cells(warp);
        // src1.f:18-23 at cell xc (0-based, right ghosts included): p -= dt (ndim-1) bulk / x_i u
        auto source = [&](real* q, int xc, double dts) {
            const double xcell = A.xlower + ((double)(xc + 1) - 0.5) * dxd;
            const double coef = dts * A.src_nd1 * A.src_bulk / xcell;
            q[0] = q[0] - (real)(coef * (double)q[ME > 1 ? 1 : 0]);
        };
        double dt = 0.0, dtdx_d = 0.0;
        // q of this lane's cell, and the interface left of it: speeds,
        // fluctuations, limited waves (src/1d/step1.f90:82, inlinelimiter)
        real q[ME], w[MW][ME], s[MW], am[ME], ap[ME];
        auto waves = [&](int b) {
            const real* rd = SMQ ? sq + b * ME * mx : A.q[b];
            real qL[ME];
#pragma unroll
            for (int m = 0; m < ME; ++m) q[m] = rd[m * fs + sx];
            if (ME > 1) q[ME > 1 ? 1 : 0] = neg ? -q[ME > 1 ? 1 : 0] : q[ME > 1 ? 1 : 0];
            if (ANY && src_split == 2 && x >= 0) source(q, x, dt / 2.0);  // Strang: dt/2 before the step
#pragma unroll
            for (int m = 0; m < ME; ++m) qL[m] = __shfl_up_sync(FULL, q[m], 1);
            A.solver.rp1(qL, q, aL, a, w, s, am, ap);
            if (order2) {
                // the waves' limiters side by side: their divisions overlap
                real ph[MW];
#pragma unroll
                for (int mw = 0; mw < MW; ++mw) {
                    real dr = real(0), nn = real(0);
#pragma unroll
                    for (int m = 0; m < ME; ++m) {
                        const real wn = __shfl_down_sync(FULL, w[mw][m], 1);
                        nn = nn + w[mw][m] * w[mw][m];
                        dr = dr + w[mw][m] * wn;
                    }
                    const real dl = __shfl_up_sync(FULL, dr, 1);
                    ph[mw] = phi_of<real>(ANY ? A.mthlim[mw] : M::lim, s[mw] > real(0) ? dl : dr, nn);
                }
#pragma unroll
                for (int mw = 0; mw < MW; ++mw) {
#pragma unroll
                    for (int m = 0; m < ME; ++m) w[mw][m] = ph[mw] * w[mw][m];
                }
            }
        };
        for (;;) {
            if (!late) waves(buf);
            __syncthreads();
            dt = sh_dt;
            dtdx_d = sh_dtdx;
            const int act = sh_act;
            if (act >= STOP_NEW) break;
            if (act == RETRY) {
                buf ^= 1;
                if (!late) waves(buf);
            }
            real* wr = SMQ ? sq + (buf ^ 1) * ME * mx : A.q[buf ^ 1];
            double c_loc = 0.0;
            for (int strip = warp; strip < nstrips; strip += nwarps) {
                if (many) cells(strip);
                if (late) waves(buf);
                real d = (real)dtdx_d, dL = d;
                if (ANY && MA > 0 && A.capa > 0) {
                    const real cap = A.capa == 1 ? a[0] : a[MAX > 1 ? 1 : 0];
                    d = (real)(dt / (dxd * (double)cap));
                    dL = __shfl_up_sync(FULL, d, 1);
                }
                if (lane >= 2 && x0 <= mx) {  // interfaces 0 .. mx
#pragma unroll
                    for (int mw = 0; mw < MW; ++mw) {  // fmax by select: a NaN leaves c_loc
                        const double cr = (double)d * (double)s[mw], cl = -(double)dL * (double)s[mw];
                        c_loc = cr > c_loc ? cr : c_loc;
                        c_loc = cl > c_loc ? cl : c_loc;
                    }
                }
                // the correction flux f, then the Godunov update and the
                // correction (src/1d/step1.f90:96-170)
                real f[ME];
                if (order2) {
                    const real ave = real(0.5) * (dL + d);
#pragma unroll
                    for (int m = 0; m < ME; ++m) f[m] = real(0);
#pragma unroll
                    for (int mw = 0; mw < MW; ++mw) {
                        const real as_ = fabs(s[mw]);
                        const real coef = ANY && A.fwave
                                              ? real(0.5) * copysign(real(1), s[mw]) * (real(1) - as_ * ave)
                                              : real(0.5) * as_ * (real(1) - as_ * ave);
#pragma unroll
                        for (int m = 0; m < ME; ++m) f[m] = f[m] + coef * w[mw][m];
                    }
                }
#pragma unroll
                for (int m = 0; m < ME; ++m) {
                    const real amr = __shfl_down_sync(FULL, am[m], 1);
                    q[m] = (q[m] - d * ap[m]) - d * amr;
                    if (order2) {
                        const real fr = __shfl_down_sync(FULL, f[m], 1);
                        q[m] = q[m] - d * (fr - f[m]);
                    }
                }
                // source after the step, before the Courant check (claw1.f:499-509)
                if (ANY && src_split != 0 && x0 >= 0) source(q, x, src_split == 2 ? dt / 2.0 : dt);
                if (lane >= 2 && lane < 2 + STRIP1 && x0 < mx) {
#pragma unroll
                    for (int m = 0; m < ME; ++m) wr[m * fs + x] = q[m];
                }
            }
            const double wm = warp_max_nonneg(c_loc > 0.0 ? c_loc : 0.0);
            if (lane == 0) red[warp] = wm;
            __syncthreads();
            buf ^= 1;
        }
        if (sh_act == STOP_OLD) buf ^= 1;
    }
    if constexpr (SMQ) {
        real* qout = A.q[cur ^ 1];
        const real* qs = sq + buf * ME * mx;
        for (int i = tid; i < ME * mx; i += blockDim.x) qout[(i / mx) * A.fstride + i % mx] = qs[i];
    }
}

}  // namespace clawb200
