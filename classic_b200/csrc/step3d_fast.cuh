// 3D unsplit step, contracted FP64 and FP32 builds (src/3d/step3.f90 with
// src/3d/flux3.f90, transverse codes of flux3.f90:189-197), for sm_100a: one
// launch per step, q and aux read once and q written once.
//
// flux3 splits, at both cells of every interface and in both directions
// across, the fluctuation and the correction flux (rpt3), and splits the
// parts again (rptt3): 24 splits per interface and sweep.  The splits of
// variable-coefficient acoustics act on the pressure part alone, with
// coefficients of the receiving cells, and every later use is linear.  With
// s = A+dq (left face) + A-dq (right face) and d = cqxx(right) - cqxx(left),
// pressure parts, a cell's share of all of them depends on two numbers per
// sweep along n:
//   X = -dt/(2 dn) s - dt/dn d          (what rpt3 splits)
//   Y = s + 3 d                         (what rptt3 splits twice)
// and the sums collapse to fluxes (K = c Z, r = 1/(Z + Z') at a face):
//   * across a face between cells a | b:  velocity r (c_b X_a + c_a X_b),
//     pressure r (K_b X_a - K_a X_b).  The y- and z-sweeps' X act on the same
//     x faces with the same factor dt/dx, so a face takes the sum of the two.
//   * at an edge with cells A B / C D around it, the double splits in both
//     orders: with f = dt^3/(6 dx dy dz), q changes by the mixed second
//     difference of f times
//       p   (m1 + m2)(Z_D yA + Z_A yD) - (m3 + m4)(Z_C yB + Z_B yC)
//       u   m1 yA + m3 yB - m4 yC - m2 yD     (along A-B)
//       v   m2 yA - m4 yB + m3 yC - m1 yD     (along A-C)
//     yA = c_D Y_A, yB = c_C Y_B, yC = c_B Y_C, yD = c_A Y_D and, with a the
//     A-C, b the B-D, g the A-B and e the C-D face's r, m1 = a e K_C,
//     m2 = b g K_B, m3 = b e K_D, m4 = a g K_A.
// 434 FP64 instructions per cell written, halo included (316 per cell computed),
// where the splits written out one by one took 1815.  The limiter works on wave strengths: the ratio of
// two waves' products is a'/a (1 + Z Z')/(1 + Z^2) with per-cell 1/(1 + Z^2).
//
// The march.  A warp holds 32 cells of a row (lane = x), a CTA ROWS rows; the
// CTA marches up z, one plane per iteration, through a segment of planes.
// x neighbours come by shuffle or from the shared planes, y neighbours
// through shared memory, z neighbours are the thread's own registers.  The
// outer two lanes and the outer row each side are halo: 28 x (ROWS-2) cells
// per plane are written.  Planes arrive by cp.async three ahead of their
// in-plane use (p, Z, c and w serve the z interfaces first).  Per plane:
//   A  strengths at the x, y and z interfaces
//   -- barrier
//   B  limited waves, correction fluxes, the x and z sums of the cell
//   -- barrier
//   C  the y sums; face fluxes of plane t, edge fluxes at plane t and
//      between planes t-1 and t
//   -- barrier
//   D  plane t-1 complete: differences of the fluxes, store
// The Courant number is the largest |c| times dt/dn in FP64, the value the
// interface-by-interface maximum takes, so the dt sequence is the
// reference-order build's.
//
// Measured against three sweep launches that formed every split (1815 FP64
// instructions and 245 B of DRAM traffic per cell): 256^3 FP64 7.45 -> 1.30
// ms per step, 161x130x147 FP32 1.02 -> 0.158.  What bounds it: FP64 at
// 192^3 runs the FP64 pipe at 30 % and issue at 50 % with 12 warps per SM
// (fixed-latency chains and the three barriers); FP32 is issue bound (71 %).
// DRAM traffic is 76 B per cell (80 algorithmic).
#pragma once
#include "char2d.cuh"
#include "step3d.cuh"

namespace clawb200 {

// Rows (warps) of a CTA and resident CTAs.  FP64: 12 rows leave 168 registers
// a thread and 8 bytes spill; the shared planes leave so little L1 that any
// spill goes to L2 (256^3, ms per step: 12 rows 1.32, 13 rows at 144
// registers 2.41, 16 rows at 128 2.1, 8 rows x 2 CTAs 1.9).  FP32: two CTAs of
// 9 rows hide each other's barriers (161x130x147, us per step, before the
// plane table: 9 x 2 167, 8 x 2 172, 10 x 2 181, 16 x 1 177, 18 x 1 188, 7 x 3
// 193).
#ifndef CLAW_STEP3F_ROWS
#define CLAW_STEP3F_ROWS 12
#endif
#ifndef CLAW_STEP3F_MINB
#define CLAW_STEP3F_MINB 1
#endif
#ifndef CLAW_STEP3F_ROWS32
#define CLAW_STEP3F_ROWS32 9
#endif
#ifndef CLAW_STEP3F_MINB32
#define CLAW_STEP3F_MINB32 2
#endif

#ifndef CLAW_STEP3F_UNROLL
#define CLAW_STEP3F_UNROLL 1  // 2 spills in FP64 (256^3: 30.1 against 24.9 ms a frame)
#endif

template <typename real>
struct Step3fShape {
    static constexpr int rows = sizeof(real) == 8 ? CLAW_STEP3F_ROWS : CLAW_STEP3F_ROWS32;
    static constexpr int minb = sizeof(real) == 8 ? CLAW_STEP3F_MINB : CLAW_STEP3F_MINB32;
    static constexpr int outx = 28, outy = rows - 2;  // cells written per plane
    static constexpr int nr = rows + 2;               // rows of a shared plane
    static constexpr int pl = nr * 32;                // values of a shared plane
    // rings: p, Z, c of 5 planes; u, v, w of 2; 20 planes that threads
    // exchange and 9 for values held from plane to plane
    static constexpr int ring = 15, uvw = 6, exch = 29;
    static constexpr int smem = (ring + uvw + exch) * pl * (int)sizeof(real);
};

template <typename real>
struct Step3fArgs {
    Sweep3Args<real> g;  // q, aux, strides, sizes, boundary conditions, method
    int tilesx, tilesy, seglen;
    const int* zrange;  // FP32: from impedance_range
};

// The exponents of n impedances: out[0] = 200 + the largest, out[1] = 200 - the
// smallest (zeroed before; 0 where there is no normal number).
__global__ void __launch_bounds__(256) impedance_range(const float* z, long long n, int* out) {
    int hi = 0, lo = 0;
    for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += gridDim.x * 256ll) {
        const int e = ((__float_as_int(z[k]) >> 23) & 255) - 127;
        if (e == -127 || e == 128) continue;
        hi = max(hi, 200 + e);
        lo = max(lo, 200 - e);
    }
    hi = __reduce_max_sync(0xffffffffu, hi);
    lo = __reduce_max_sync(0xffffffffu, lo);
    if ((threadIdx.x & 31) == 0 && hi > 0) {
        atomicMax(out, hi);
        atomicMax(out + 1, lo);
    }
}

// Where a plane's q and aux lie in global memory, and whether w changes its sign
// (1) or takes the piston's (2) there.
template <typename real>
struct Plane3f {
    const real *q, *aux;
    int w;
};

// zt holds planes t-1 .. t+4 at [pos & 7].  One thread fills an entry a plane
// ahead; each thread for itself, three times a plane, it cost the FP32 kernel,
// bound by issue, 5 % (192^3 314 -> 298 us a step; FP64 517 -> 509).
// UNIT: the grid takes 2^e as its unit of impedance and pressure.
template <typename real, int LIM, bool TRANS, bool UNIT>
__device__ __forceinline__ void step3f_march(const Step3fArgs<real>& A, const StepHead& hd, unsigned char* smem_raw,
                                             double* red, Plane3f<real>* zt, int e) {
    using Sh = Step3fShape<real>;
    constexpr int ROWS = Sh::rows, PL = Sh::pl;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int kUnroll = CLAW_STEP3F_UNROLL;
    const Sweep3Args<real>& a = A.g;
    ClawCtl* ctl = a.ctl;
    const double tbc = *(volatile double*)&ctl->told;
    const int cur = hd.cur;
    const double dt = hd.dt;
    const real* __restrict__ qold = a.q[cur];
    real* __restrict__ qnew = a.q[cur ^ 1];
    const real* __restrict__ aux = a.aux;
    const real tx = (real)(dt / a.d[0]), ty = (real)(dt / a.d[1]), tz = (real)(dt / a.d[2]);
    const real half2 = a.order == 2 ? real(0.5) : real(0);   // order 1: no correction fluxes
    const real xd = a.m3 == 2 ? real(1) : real(0);           // rpt3 splits the correction flux too
    const real yd = a.m3 == 2 && a.m4 == 2 ? real(3) : real(0);
    const real f6 = TRANS && a.m4 > 0 ? (real(1) / real(6)) * tx * ty * tz : real(0);
    const int lim1 = a.mthlim[0], lim2 = a.mthlim[1];

    const int mx = a.m[0], my = a.m[1], mz = a.m[2];
    const int lane = threadIdx.x & 31;
    // FP32, bound by issue: a warp-uniform value to the compiler (3 % faster);
    // in FP64 that costs registers it does not have
    const int r = sizeof(real) == 4 ? __shfl_sync(FULL, (int)(threadIdx.x >> 5), 0) : (int)(threadIdx.x >> 5);
    int bid = blockIdx.x;
    const int bx = bid % A.tilesx;
    bid /= A.tilesx;
    const int by = bid % A.tilesy, seg = bid / A.tilesy;
    const int k0 = 1 + seg * A.seglen, k1 = min(k0 + A.seglen, mz + 1);  // planes written: k0 .. k1-1
    const int i = 1 + bx * Sh::outx - 2 + lane;  // this thread's column
    const int j0 = 1 + by * Sh::outy;            // first row written
    const int j = j0 - 1 + r;                    // this warp's row
    const bool out = lane >= 2 && lane < 30 && i <= mx && r >= 1 && r < ROWS - 1 && j <= my;

    // zu takes Z and pressure differences into the unit, pu takes pressure
    // increments out of it, `one` is the 1 that u's part has beside Z Z'
    // (negligible, or all there is, where the bound takes effect)
    real zu = real(1), pu = real(1), one = real(1);
    if constexpr (UNIT) {
        zu = __int_as_float((127 - e) << 23);
        pu = __int_as_float((127 + e) << 23);
        one = fminf(zu * zu, 0x1p100f);
    }
    const real txp = UNIT ? tx * pu : tx, typ = UNIT ? ty * pu : ty, tzp = UNIT ? tz * pu : tz;
    auto pdiff = [&](real x, real y) { return UNIT ? (x - y) * zu : x - y; };

    // source cell of a column and a row under the boundary conditions; cells
    // past the last ghost layer repeat it (nothing written depends on them)
    bool negx, negy, negb, negh;
    const int ic = min(i, mx + 2), jc = min(j, my + 2);
    const int im = bc3_src(ic, mx, a.bc[0], a.bc[1], negx);
    const int jm = bc3_src(jc, my, a.bc[2], a.bc[3], negy);
    (void)bc3_src(min(j - 1, my + 2), my, a.bc[2], a.bc[3], negb);  // the row below
    // the first and the last warp also copy the row beyond theirs
    const bool edge = r == 0 || r == ROWS - 1;
    const int jh = min(r == 0 ? j - 1 : j + 1, my + 2);
    const int jhm = bc3_src(jh, my, a.bc[2], a.bc[3], negh);
    const long long qxy = (long long)(im - 1) + (long long)(jm - 1) * a.qs[1];
    const long long qxh = (long long)(im - 1) + (long long)(jhm - 1) * a.qs[1];
    const long long axy = (long long)(ic + 1) + (long long)(jc + 1) * a.as[1];
    const long long axh = (long long)(ic + 1) + (long long)(jh + 1) * a.as[1];

    real* ring = reinterpret_cast<real*>(smem_raw);  // [5][p, Z, c][PL]
    real* uvw = ring + Sh::ring * PL;                // [2][u, v, w][PL]
    real* ex = uvw + Sh::uvw * PL;
    const int own = (r + 1) * 32 + lane;
    const int lm = own - (lane > 0 ? 1 : 0), lp = own + (lane < 31 ? 1 : 0);
    const int hal = r == 0 ? lane : (ROWS + 1) * 32 + lane;
    real *SA1 = ex, *SA2 = ex + PL, *SG = ex + 2 * PL, *ST1 = ex + 3 * PL, *SCP = ex + 4 * PL,
         *SCV = ex + 5 * PL, *SXY = ex + 6 * PL, *SYZ = ex + 7 * PL, *SRZ = ex + 8 * PL;
    real* SP = ex + 9 * PL;    // [2 by the plane's parity][Yx, rx, ry]
    real* SE = ex + 15 * PL;   // [5] what a row hands to the row above it
    // [9] values held from plane to plane (registers would spill): plane t-1's
    // q plus its own sums, the edge fluxes at t-3/2, plane t-1's Yy
    real* SB = ex + 20 * PL;

    auto fill = [&](int pos) {
        bool neg;
        const int pm = bc3_src(min(pos, mz + 2), mz, a.bc[4], a.bc[5], neg);
        zt[pos & 7].q = qold + (long long)(pm - 1) * a.qs[2];
        zt[pos & 7].aux = aux + (long long)(min(pos, mz + 2) + 1) * a.as[2];
        zt[pos & 7].w = (neg ? 1 : 0) | (pos > mz && a.bc[5] == BC_PISTON ? 2 : 0);
    };
    // copies of plane pos: p, Z, c into ring slot `so`, w into its parity's
    auto issue_pzc = [&](int pos, int so) {
        const real *q = zt[pos & 7].q, *x = zt[pos & 7].aux;
        real* d = ring + so + own;
        cp_async_el(d, q + qxy);
        cp_async_el(d + PL, x + axy);
        cp_async_el(d + 2 * PL, x + axy + a.afstride);
        cp_async_el(uvw + ((pos & 1) * 3 + 2) * PL + own, q + qxy + 3 * a.fstride);
        if (edge) {
            real* h = ring + so + hal;
            cp_async_el(h, q + qxh);
            cp_async_el(h + PL, x + axh);
            cp_async_el(h + 2 * PL, x + axh + a.afstride);
        }
    };
    auto issue_uv = [&](int pos) {
        const real* q = zt[pos & 7].q;
        real* d = uvw + (pos & 1) * 3 * PL;
        cp_async_el(d + own, q + qxy + a.fstride);
        cp_async_el(d + PL + own, q + qxy + 2 * a.fstride);
        if (edge) cp_async_el(d + PL + hal, q + qxh + 2 * a.fstride);
    };
    // own Z's of a landed plane into the unit (before the barrier that publishes them)
    auto to_unit = [&](int so) {
        if (UNIT) {
            ring[so + PL + own] *= zu;
            if (edge) ring[so + PL + hal] *= zu;
        }
    };
    // w at plane pos from its stored value (the walls' and the piston's sign)
    auto wbc = [&](int pos, real w) {
        const int f = zt[pos & 7].w;
        if (f & 1) w = -w;
        if (f & 2) w = (real)(2.0 * piston_speed(a, i, j, tbc)) - w;
        return w;
    };
    auto lim_a = [&](real s, real n) { return limited_strength<real, LIM, true>(s, n, lim1); };
    auto lim_b = [&](real s, real n) { return limited_strength<real, LIM, true>(s, n, lim2); };
    // factor of a limited wave in the correction flux of a direction: |s| (1 - |s| dt/dn) / 2
    auto coef = [&](real c, real tn) { return half2 * fabs(c) * (real(1) - fabs(c) * tn); };
    // p, u (along A-B) and v (along A-C) of an edge flux
    auto edge_flux = [&](real ra, real rb, real rg, real re, real zA, real cA, real zB, real cB, real zC,
                         real cC, real zD, real cD, real YA, real YB, real YC, real YD, real& ep,
                         real& eu, real& ev) {
        const real m1 = (ra * re) * (cC * zC), m2 = (rb * rg) * (cB * zB);
        const real m3 = (rb * re) * (cD * zD), m4 = (ra * rg) * (cA * zA);
        const real yA = cD * YA, yB = cC * YB, yC = cB * YC, yD = cA * YD;
        ep = (m1 + m2) * (zD * yA + zA * yD) - (m3 + m4) * (zC * yB + zB * yC);
        eu = (m1 * yA - m2 * yD) + (m3 * yB - m4 * yC);
        ev = (m2 * yA - m1 * yD) + (m3 * yC - m4 * yB);
    };

    // ---- planes t0-1 .. t0+2 (t0 = k0 - 1): z strengths at t0-1/2 and t0+1/2
    int sm = 0, s0 = 3 * PL, s1 = 6 * PL, s2 = 9 * PL, s3 = 12 * PL;  // slots of planes t-1 .. t+3
    const int t0 = k0 - 1;
    real w0, w1, wm;  // w at planes t, t+1 (t-1)
    real a1z, a2z, a2zm, rz, rz1, g0;
    if (threadIdx.x < 6) fill(t0 - 1 + (int)threadIdx.x);
    __syncthreads();
    {
        auto w_at = [&](int pos) { return wbc(pos, zt[pos & 7].q[qxy + 3 * a.fstride]); };
        wm = w_at(t0 - 1);
        w0 = w_at(t0);
        w1 = w_at(t0 + 1);
    }
    issue_pzc(t0 - 1, sm);
    issue_pzc(t0, s0);
    issue_uv(t0);
    // the w copies of planes t0-1 and t0 must not land after those of t0+1 and t0+2
    cp_async_wait_all();
    to_unit(sm);
    to_unit(s0);
    __syncthreads();
    issue_pzc(t0 + 1, s1);
    issue_pzc(t0 + 2, s2);
    cp_async_wait_all();
    to_unit(s1);
    to_unit(s2);
    __syncthreads();
    {
        const real pA = ring[sm + own], zA = ring[sm + PL + own];
        const real pB = ring[s0 + own], zB = ring[s0 + PL + own];
        const real pC = ring[s1 + own], zC = ring[s1 + PL + own];
        rz = rcp_newton(zA + zB);
        rz1 = rcp_newton(zB + zC);
        a2zm = (zA * (w0 - wm) + pdiff(pB, pA)) * rz;
        a1z = (zC * (w1 - w0) - pdiff(pC, pB)) * rz1;
        a2z = (zB * (w1 - w0) + pdiff(pC, pB)) * rz1;
        g0 = rcp_newton(one + zB * zB);
    }
    real t2zm = 0, cpzm = 0, cwzm = 0;          // z interface t-1/2: right-going fluctuation, correction flux
    real cmax = 0;
    real fxp = 0, fxu = 0, fyp = 0, fyv = 0;    // plane t-1: face fluxes so far
    real fzp = 0, fzw = 0;                      // z face t-3/2
    real XZm = 0;                               // plane t-1
    const bool inxy = i >= 0 && i <= mx + 1 && j <= my + 1 && lane >= 1;

#pragma unroll kUnroll
    for (int t = t0; t <= k1; ++t) {
        if (t + 3 <= k1 + 1) issue_pzc(t + 3, s3);
        if (t + 1 <= k1) issue_uv(t + 1);
        if (threadIdx.x == 0) fill(t + 4);
        const int par = t & 1;
        real* SPt = SP + par * 3 * PL;
        real* SPm = SP + (par ^ 1) * 3 * PL;
        // ------------------------------------------------- A: strengths
        const real* P = ring + s0;
        const real p = P[own], z = P[PL + own], c = P[2 * PL + own];
        const real* UV = uvw + par * 3 * PL;
        real u = UV[own], v = UV[PL + own];
        if (negx) u = -u;
        if (negy) v = -v;
        if (inxy && fabs(c) > cmax) cmax = fabs(c);  // a NaN leaves it
        const real zl = P[PL + lm], cl = P[2 * PL + lm];
        real rx, a1x, a2x;
        {
            const real du = u - __shfl_up_sync(FULL, u, 1), dp = pdiff(p, P[lm]);
            rx = rcp_newton(zl + z);
            a1x = (z * du - dp) * rx;
            a2x = (zl * du + dp) * rx;
        }
        const real zb = P[PL + own - 32], cb = P[2 * PL + own - 32];
        real ry, a1y, a2y;
        {
            real vb = UV[PL + own - 32];
            if (negb) vb = -vb;
            const real dv = v - vb, dp = pdiff(p, P[own - 32]);
            ry = rcp_newton(zb + z);
            a1y = (z * dv - dp) * ry;
            a2y = (zb * dv + dp) * ry;
        }
        SA1[own] = a1y;
        SA2[own] = a2y;
        SG[own] = g0;
        SRZ[own] = rz;
        SPt[PL + own] = rx;
        SPt[2 * PL + own] = ry;
        if (r == ROWS - 1) {  // the left-going strength one row above, and that face's r
            real va = UV[PL + own + 32];
            if (negh) va = -va;
            const real za = P[PL + own + 32];
            SA1[own + 32] = (za * (va - v) - pdiff(P[own + 32], p)) * rcp_newton(z + za);
        }
        // z interface t+3/2
        const real z1 = ring[s1 + PL + own], c1 = ring[s1 + 2 * PL + own];
        const real z2 = ring[s2 + PL + own];
        const real w2 = wbc(t + 2, uvw[(par * 3 + 2) * PL + own]);
        real a1zn, a2zn, rz2;
        {
            const real dw = w2 - w1, dp = pdiff(ring[s2 + own], ring[s1 + own]);
            rz2 = rcp_newton(z1 + z2);
            a1zn = (z2 * dw - dp) * rz2;
            a2zn = (z1 * dw + dp) * rz2;
        }
        const real g1 = rcp_newton(one + z1 * z1);
        __syncthreads();
        // ---------------------------- B: limited waves, x and z sums
        real bp = p, bu = u, bv = v, bw = w0;
        real Xx, Yx, Xz, Yz;
        {
            const real h = one + zl * z;
            const real n1 = __shfl_down_sync(FULL, a1x, 1) * (h * __shfl_up_sync(FULL, g0, 1));
            const real n2 = __shfl_up_sync(FULL, a2x, 1) * (h * g0);
            const real e1 = coef(cl, tx) * lim_a(a1x, n1), e2 = coef(c, tx) * lim_b(a2x, n2);
            const real cp = z * e2 - zl * e1, cu = e1 + e2;
            const real ta = cl * a1x, tb = c * a2x;
            const real tr = __shfl_down_sync(FULL, ta, 1);
            const real sp = z * (tb + tr), su = tb - tr;
            const real dp = __shfl_down_sync(FULL, cp, 1) - cp, du = __shfl_down_sync(FULL, cu, 1) - cu;
            bp -= txp * (sp + dp);
            bu -= tx * (su + du);
            Xx = -tx * (real(0.5) * sp + xd * dp);
            Yx = sp + yd * dp;
        }
        {
            const real h = one + z * z1;
            const real e1 = coef(c, tz) * lim_a(a1z, a1zn * (h * g0));
            const real e2 = coef(c1, tz) * lim_b(a2z, a2zm * (h * g1));
            const real cp = z1 * e2 - z * e1, cw = e1 + e2;
            const real ta = c * a1z;
            const real sp = z * (t2zm + ta), sw = t2zm - ta;
            const real dp = cp - cpzm, dw = cw - cwzm;
            bp -= tzp * (sp + dp);
            bw -= tz * (sw + dw);
            Xz = -tz * (real(0.5) * sp + xd * dp);
            Yz = sp + yd * dp;
            t2zm = c1 * a2z;
            cpzm = cp;
            cwzm = cw;
        }
        real cpy = 0, cvy = 0, tby = 0;
        if (r >= 1) {  // y interface below this row
            const real h = one + zb * z;
            const real n1 = SA1[own + 32] * (h * SG[own - 32]);
            const real n2 = SA2[own - 32] * (h * g0);
            const real e1 = coef(cb, ty) * lim_a(a1y, n1), e2 = coef(c, ty) * lim_b(a2y, n2);
            cpy = z * e2 - zb * e1;
            cvy = e1 + e2;
            tby = c * a2y;
            ST1[own] = cb * a1y;
            SCP[own] = cpy;
            SCV[own] = cvy;
        }
        if (TRANS) {
            SXY[own] = Xx + Xz;
            SYZ[own] = Yz;
            SPt[own] = Yx;
        }
        __syncthreads();
        // ------------- C: y sums, fluxes at plane t and at z face t-1/2
        real Xy = 0, Yy = 0;
        if (r >= 1 && r < ROWS - 1) {
            const real tr = ST1[own + 32];
            const real sp = z * (tby + tr), sv = tby - tr;
            const real dp = SCP[own + 32] - cpy, dv = SCV[own + 32] - cvy;
            bp -= typ * (sp + dp);
            bv -= ty * (sv + dv);
            Xy = -ty * (real(0.5) * sp + xd * dp);
            Yy = sp + yd * dp;
        }
        real nfxp = 0, nfxu = 0, nfyp = 0, nfyv = 0, nfzp = 0, nfzw = 0;
        real nexzp = 0, nexzu = 0, exzw = 0, neyzp = 0, neyzv = 0, eyzw = 0, exyp = 0, exyu = 0, exyv = 0;
        const real XX = Xy + Xz, XZ = Xx + Xy;
        if (TRANS && r < ROWS - 1) {
            const real* M = ring + sm;  // plane t-1
            const real zR = P[PL + lp], cR = P[2 * PL + lp];
            const real zU = P[PL + own + 32], cU = P[2 * PL + own + 32];
            const real rxR = SPt[PL + lp], ryU = SPt[2 * PL + own + 32];
            const real zm = M[PL + own], cm = M[2 * PL + own];
            {  // faces i+1/2, j+1/2, t-1/2
                const real XR = __shfl_down_sync(FULL, XX, 1);
                const real hi = cR * (rxR * XX), lo = c * (rxR * XR);
                nfxu = tx * (hi + lo);
                nfxp = tx * (zR * hi - z * lo);
                const real hu = cU * (ryU * (Xx + Xz)), lu = c * (ryU * SXY[own + 32]);
                nfyv = ty * (hu + lu);
                nfyp = ty * (zU * hu - z * lu);
                const real hz = c * (rz * XZm), lz = cm * (rz * XZ);
                nfzw = tz * (hz + lz);
                nfzp = tz * (z * hz - zm * lz);
            }
            {  // edge (i+1/2, j+1/2) of plane t
                const real zD = P[PL + lp + 32], cD = P[2 * PL + lp + 32];
                edge_flux(ryU, SPt[2 * PL + lp + 32], rxR, SPt[PL + lp + 32], z, c, zR, cR, zU, cU, zD, cD, Yz,
                          SYZ[lp], SYZ[own + 32], SYZ[lp + 32], exyp, exyu, exyv);
            }
            {  // edge (i+1/2, t-1/2)
                const real YR = __shfl_down_sync(FULL, Yy, 1);
                edge_flux(rz, SRZ[lp], SPm[PL + lp], rxR, zm, cm, M[PL + lp], M[2 * PL + lp], z, c, zR, cR,
                          SB[8 * PL + own], SB[8 * PL + lp], Yy, YR, nexzp, nexzu, exzw);
            }
            {  // edge (j+1/2, t-1/2)
                edge_flux(rz, SRZ[own + 32], SPm[2 * PL + own + 32], ryU, zm, cm, M[PL + own + 32],
                          M[2 * PL + own + 32], z, c, zU, cU, SPm[own], SPm[own + 32], Yx, SPt[own + 32], neyzp,
                          neyzv, eyzw);
            }
            // the y faces of plane t-1 are complete
            fyp += f6 * (neyzp - SB[6 * PL + own]);
            fyv += f6 * (neyzv - SB[7 * PL + own]);
            SB[6 * PL + own] = neyzp;
            SB[7 * PL + own] = neyzv;
            SE[own] = fyp;
            SE[PL + own] = fyv;
            SE[2 * PL + own] = eyzw;
            SE[3 * PL + own] = exyp;
            SE[4 * PL + own] = exyu;
        }
        cp_async_wait_all();
        if (t + 3 <= k1 + 1) to_unit(s3);
        __syncthreads();
        // -------------------------------------------- D: plane t-1
        real op = SB[own], ou = SB[PL + own], ov = SB[2 * PL + own], ow = SB[3 * PL + own];
        SB[own] = bp;
        SB[PL + own] = bu;
        SB[2 * PL + own] = bv;
        SB[3 * PL + own] = bw;
        if (TRANS && r >= 1 && r < ROWS - 1) {
            fxp += f6 * (nexzp - SB[4 * PL + own]);
            fxu += f6 * (nexzu - SB[5 * PL + own]);
            SB[4 * PL + own] = nexzp;
            SB[5 * PL + own] = nexzu;
            nfzw += f6 * ((exzw - __shfl_up_sync(FULL, exzw, 1)) + (eyzw - SE[2 * PL + own - 32]));
            const real dfp = ((fxp - __shfl_up_sync(FULL, fxp, 1)) + (fyp - SE[own - 32])) + (nfzp - fzp);
            op -= UNIT ? pu * dfp : dfp;
            ou -= fxu - __shfl_up_sync(FULL, fxu, 1);
            ov -= fyv - SE[PL + own - 32];
            ow -= nfzw - fzw;
            // plane t's x faces take the y difference of its edge fluxes
            fxp = nfxp + f6 * (exyp - SE[3 * PL + own - 32]);
            fxu = nfxu + f6 * (exyu - SE[4 * PL + own - 32]);
        }
        if (TRANS) {
            fyp = nfyp;
            fyv = nfyv + f6 * (exyv - __shfl_up_sync(FULL, exyv, 1));  // ... and its y faces the x difference
            fzp = nfzp;
            fzw = nfzw;
            XZm = XZ;
            SB[8 * PL + own] = Yy;
        }
        if (out && t > k0) {
            const long long o = (long long)(i - 1) + (long long)(j - 1) * a.qs[1] + (long long)(t - 2) * a.qs[2];
            qnew[o] = op;
            qnew[o + a.fstride] = ou;
            qnew[o + 2 * a.fstride] = ov;
            qnew[o + 3 * a.fstride] = ow;
        }
        w0 = w1;
        w1 = w2;
        a2zm = a2z;
        a1z = a1zn;
        a2z = a2zn;
        rz = rz1;
        rz1 = rz2;
        g0 = g1;
        const int so = sm;
        sm = s0;
        s0 = s1;
        s1 = s2;
        s2 = s3;
        s3 = so;
    }
    const double cd = (double)cmax;
    const double cfl = fmax(fmax(sweep_cfl(dt / a.d[0], cd), sweep_cfl(dt / a.d[1], cd)), sweep_cfl(dt / a.d[2], cd));
    cta_cfl_and_control(ctl, cfl, red);
}

template <typename real, int LIM, bool TRANS>
__global__ void __launch_bounds__(32 * Step3fShape<real>::rows, Step3fShape<real>::minb)
step3f_kernel(const __grid_constant__ Step3fArgs<real> A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[Step3fShape<real>::rows];
    __shared__ Plane3f<real> zt[8];
    grid_dependency_sync();
    const StepHead hd = step_head(A.g.ctl);
    if (hd.done) return;
    // FP32: products of impedances (1 + Z Z', r r' K) leave its range beyond Z =
    // 2^+-62.  A grid with some Z beyond 2^+-40 takes the power of two amid its
    // Z's as unit of impedance and pressure, which changes exponents only.  A
    // march of its own: the few multiplications cost the others 2.8 %
    // (161x130x147 1426 -> 1466 us a frame).
    if constexpr (sizeof(real) == 4) {
        const int hi = A.zrange[0] - 200, lo = 200 - A.zrange[1];
        const int e = max(-126, min(126, (hi + lo) / 2));
        if (hi > -200 && (hi > 40 || lo < -40) && e != 0) {
            step3f_march<real, LIM, TRANS, true>(A, hd, smem_raw, red, zt, e);
            return;
        }
    }
    step3f_march<real, LIM, TRANS, false>(A, hd, smem_raw, red, zt, 0);
}

}  // namespace clawb200
