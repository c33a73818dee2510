// 3D unsplit wave-propagation step (src/3d/step3.f90:3-873 with
// src/3d/flux3.f90:4-612) for sm_100a.
//
// One kernel per sweep direction.  A CTA owns a T3A x T3B tile of slices of
// that sweep (the outer ring of the tile is a one-slice halo) and marches the
// tile along the slice direction, one cell position per iteration; each slice's
// Riemann state (normal solve at interface p+2, limiter and second-order
// correction at p+1, the transverse and double-transverse splits of p+1, and
// the gadd/hadd partial sums of cells p and p+1) is carried by a pair of
// threads, the same lane of two neighbouring warps.
//
// A cell receives contributions from the nine slices around it.  step3 adds
// them in the order of its 2x2-block colouring (colour of the slow slice
// index, colour of the fast one, then slow, then fast index), which fixes the
// rounding of every cell.  Here each slice publishes the terms it adds to its
// eight neighbours in shared memory and every cell adds its nine terms in
// that same order, so the x-, y- and z-sweeps reproduce the serial loop nest
// bit for bit; the three sweeps run as three launches in step3's order.
//
// q is stored for interior cells only; ghost values come from the boundary
// conditions of bc3 (x pass, then y, then z, so corners compose the maps).
#pragma once
#include "common.cuh"
#include "riemann.cuh"

namespace clawb200 {

#ifndef CLAW_T3B
#define CLAW_T3B 12
#endif
#ifndef CLAW_SWEEP3_MINB
#define CLAW_SWEEP3_MINB 1  // resident CTAs per SM the sweep kernels are compiled for
#endif
constexpr int T3A = 16, T3B = CLAW_T3B, NT3 = T3A * T3B;   // thread tile, incl. the halo ring
constexpr int S3A = T3A + 2, S3B = T3B + 2, NS3 = S3A * S3B;  // aux tile, one more ring
constexpr int RING3 = 4;                              // aux positions held in shared memory
constexpr int NPL3 = 4;                               // aux planes: Z, c, 1/(Z+Z_e1), 1/(Z+Z_e2)
constexpr int NTERM3 = 39;                            // terms per slice and position: 8 neighbours x 4, centre
constexpr int BC_PISTON = 10;                         // user BC of acoustics_3d_heterogeneous

template <typename real>
struct Sweep3Args {
    real* q[2];
    const real* aux;
    long long qs[3];     // q strides in elements along x, y, z (1, ld, ld*my)
    long long fstride;   // q field pitch
    long long as[3];     // aux strides (1, ald, ald*(my+4))
    long long afstride;  // aux field pitch
    int m[3];            // mx, my, mz
    int bc[6];           // [2*axis + side]: mthbc
    int mthlim[2];
    int order, m3, m4;
    double d[3];         // dx, dy, dz
    double xlower, ylower;
    int tilesA, tilesB, nseg, seglen;
    ClawCtl* ctl;
};

constexpr int QST3 = 4;  // staged q planes of NT3 values: [position & 1][p, normal velocity]

constexpr int XCH3 = 8;   // exchange planes of NT3 values: L [h][2], R [h][2]
constexpr int VST3 = 8;   // staged values of the cells each role updates: [position & 1][role][2]

// Shared memory is sized to the carveout steps (100, 132, 164, 196, 228 KB);
// what the carveout leaves is L1, which serves the x-sweep's strided loads and
// the spills: 121 KB with one buffer of terms (a second CTA barrier a position).
template <typename real>
__host__ __device__ constexpr int sweep3_smem_bytes() {
    return (RING3 * NPL3 * NS3 + (NTERM3 + XCH3 + QST3 + VST3) * NT3) * (int)sizeof(real) +
           16 * (int)sizeof(double);
}

// one element global -> shared, asynchronously (cp.async, 4 or 8 bytes)
template <typename real>
__device__ __forceinline__ void cp_async_el(real* dst, const real* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "n"((int)sizeof(real))
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Source index of (possibly ghost) cell idx along an axis of n cells, and
// whether a solid wall negates the normal velocity (src/3d/bc3.f).
__device__ __forceinline__ int bc3_src(int idx, int n, int lo, int hi, bool& flip) {
    flip = false;
    if (idx < 1) {
        if (lo == BC_PERIODIC) return idx + n;
        if (lo == BC_EXTRAP) return 1;
        flip = (lo == BC_WALL);
        return 1 - idx;
    }
    if (idx > n) {
        if (hi == BC_PERIODIC) return idx - n;
        if (hi == BC_EXTRAP) return n;
        flip = (hi == BC_WALL);
        return 2 * n + 1 - idx;  // wall and piston reflect
    }
    return idx;
}

// Piston velocity of examples/acoustics_3d_heterogeneous/bc3.f:296-309 at the
// ghost column (i, j) and time t: s = -exp(-500 r^2) exp(-500 t^2) for t < 0.1,
// flushed to 0 below 1e-6 in magnitude.
__device__ __forceinline__ double piston_speed(const Sweep3Args<double>& a, int i, int j, double t) {
    if (!(t < 0.1)) return 0.0;
    const double xi = a.xlower + ((double)i - 0.5) * a.d[0];
    const double yj = a.ylower + ((double)j - 0.5) * a.d[1];
    const double r2 = xi * xi + yj * yj;
    double s = -(exp(-(500.0 * r2)) * exp(-(500.0 * (t * t))));
    if (fabs(s) < 1e-6) s = 0.0;
    return s;
}
__device__ __forceinline__ double piston_speed(const Sweep3Args<float>& a, int i, int j, double t) {
    Sweep3Args<double> b;
    b.xlower = a.xlower; b.ylower = a.ylower; b.d[0] = a.d[0]; b.d[1] = a.d[1];
    return piston_speed(b, i, j, t);
}

// flux3's method split (src/3d/flux3.f90:189-197) as compile-time values when
// known (-1: read from the arguments).
template <int M3, int M4, int LIM>
struct Method3D {
    static constexpr int m3 = M3, m4 = M4, lim = LIM;
};
using MethodGeneric3D = Method3D<-1, -1, -1>;
using MethodMC3D = Method3D<2, 2, 4>;  // transverse_waves 22, MC on both waves

constexpr int NT3P = 2 * NT3;

// the quotients outside quot_rcp's range, out of line: they hardly ever run
template <class S>
__device__ __noinline__ typename S::Split split3_far(typename S::real xp, typename S::real zb, typename S::real cb,
                                                     typename S::real zm, typename S::real za,
                                                     typename S::real ca) {
    return S::split(xp, zb, cb, zm, za, ca);
}

// Role h = 0 owns flux3's y-like side (the rpt3 splits in e1, the rptt3 splits
// of the z-like parts in e1, gadd), h = 1 the z-like side (splits in e2, hadd);
// both solve the normal problem, limit and form cqxx (a few dozen operations,
// duplicated).  A warp's role is a compile-time constant, so shared-memory
// indexes fold to immediates.  The four combinations each side needs from the
// other's splits (flux3.f90:363-376 and :488-495) cross through shared memory
// under a 64-thread named barrier of the warp pair.  Operation order per value
// is flux3's.
//
// A cell adds its terms in step3's colour order, which depends on its slice
// indexes modulo 4: each thread sorts its neighbours once and keeps the shared
// memory offsets of its terms in that order, the centre's own terms among them
// (published like the neighbours'), so the gather is a run of loads and adds.
//
// The four rpt3 splits of a position, and the four rptt3 splits after the
// exchange, are formed side by side so that their quotients overlap.
//
// Against pairs of neighbouring lanes with run-time roles, an IEEE division in
// every quotient, the gather's indexes formed at every position and segments
// of 64 cells whatever the grid, ms a step: 256^3 15.1 -> 11.0, 128^3 3.0 ->
// 1.69, 64^3 1.53 -> 0.25.  99 warp instructions a cell and sweep for 151; the
// FP64 pipe runs at 27 %, latency of dependent FP64 operations bounds it.
__device__ __forceinline__ void pair_sync(int id) {
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}

// The march of one tile of slices for the threads of role H; returns the
// thread's Courant number.
template <class S, int DIR, class M, int H>
__device__ __forceinline__ double sweep3p_march(const Sweep3Args<typename S::real>& a,
                                                unsigned char* smem_raw, int* far) {
    using real = typename S::real;
    using Split = typename S::Split;
    constexpr int AXN = DIR, AXA = DIR == 0 ? 1 : 0, AXB = DIR == 2 ? 1 : 2;
    constexpr bool E1A = DIR != 1;
    constexpr int CN = 1 + AXN, CE1 = 1 + (E1A ? AXA : AXB), CE2 = 1 + (E1A ? AXB : AXA);
    constexpr int NPL = NPL3;
    // shared-memory steps of this role's own split direction and the other
    constexpr int E1S = E1A ? 1 : S3A, E2S = E1A ? S3A : 1;
    constexpr int OWNS = H ? E2S : E1S, OTHS = H ? E1S : E2S;
    constexpr int CA = H ? CE1 : 0, CB = H ? CE2 : CN;  // components this role updates

    real* saux = reinterpret_cast<real*>(smem_raw);  // [RING3][NPL][NS3]
    real* sterm = saux + RING3 * NPL * NS3;          // [NTERM3][NT3]
    real* sxch = sterm + NTERM3 * NT3;               // [XCH3][NT3]
    real* sq = sxch + XCH3 * NT3;                    // [QST3][NT3]
    real* sv = sq + QST3 * NT3;                      // [VST3][NT3]

    ClawCtl* ctl = a.ctl;
    const int cur = ctl->cur;
    const real* __restrict__ qold = a.q[cur];
    real* __restrict__ qnew = a.q[cur ^ 1];
    const real* __restrict__ aux = a.aux;
    const double dt = ctl->dt;
    const double tbc = ctl->told;
    const double tn_d = dt / a.d[AXN];
    const real tn = (real)tn_d;
    const real te1 = (real)(dt / a.d[E1A ? AXA : AXB]);
    const real te2 = (real)(dt / a.d[E1A ? AXB : AXA]);
    const real H5 = real(0.5) * tn;
    const real S6g = (real(1.0) / real(6.0)) * tn * te2;
    const real S6h = (real(1.0) / real(6.0)) * tn * te1;
    const real dtdxave = real(0.5) * (tn + tn);
    const real t_own = H ? te2 : te1;
    const real S6own = H ? S6h : S6g;

    const int m3 = M::m3 >= 0 ? M::m3 : a.m3;
    const int m4 = M::m4 >= 0 ? M::m4 : a.m4;
    const int order = M::m3 >= 0 ? 2 : a.order;

    const int mN = a.m[AXN], mA = a.m[AXA], mB = a.m[AXB];
    const int bid = blockIdx.x;
    const int seg = bid % a.nseg, tile = bid / a.nseg;
    const int A0 = 1 + (tile % a.tilesA) * (T3A - 2);
    const int B0 = 1 + (tile / a.tilesA) * (T3B - 2);
    const int p0 = 1 + seg * a.seglen;
    const int p1 = min(p0 + a.seglen, mN + 1);
    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int sl = (warp >> 1) * 32 + (tid & 31);  // slice within the tile
    const int pair_id = 1 + (warp >> 1);           // named barrier of the warp pair
    const int ta = sl % T3A, tb = sl / T3A;
    const int A = A0 - 1 + ta, B = B0 - 1 + tb;
    const bool active = A <= mA + 1 && B <= mB + 1;
    const bool apply = active && ta >= 1 && ta <= T3A - 2 && tb >= 1 && tb <= T3B - 2 &&
                       A <= mA && B <= mB;

    // step3's order of the cell's nine contributions (src/3d/step3.f90:151-186:
    // colour of the slow slice index, colour of the fast one, slow, fast), as
    // offsets into the published terms: planes off and off + 2.  Role 0's
    // centre is two entries, (own sums) and (the transverse differences).
    constexpr int NG = H ? 9 : 10;
    int goff[NG];
    {
        unsigned long long perm = 0;
        int code[9], key[9];
        for (int k = 0; k < 9; ++k) {
            const int da = k % 3 - 1, db = k / 3 - 1;
            const int sA = A + da, sB = B + db;
            code[k] = k;
            key[k] = (((sB >> 1) & 1) << 5) | (((sA >> 1) & 1) << 4) | ((db + 1) << 2) | (da + 1);
        }
        for (int i = 1; i < 9; ++i)
            for (int j = i; j > 0 && key[j - 1] > key[j]; --j) {
                int t = key[j]; key[j] = key[j - 1]; key[j - 1] = t;
                t = code[j]; code[j] = code[j - 1]; code[j - 1] = t;
            }
        int kc = 0;  // place of the centre
        for (int k = 0; k < 9; ++k) {
            perm |= (unsigned long long)code[k] << (4 * k);
            if (code[k] == 4) kc = k;
        }
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int k = H == 0 && g > kc ? g - 1 : g;
            const int cd = (int)((perm >> (4 * k)) & 15ull);
            const int da = cd % 3 - 1, db = cd / 3 - 1;
            const int u = E1A ? -da : -db, w = E1A ? -db : -da;
            const int idx9 = (w + 1) * 3 + (u + 1);
            const int nb = idx9 < 4 ? idx9 : idx9 - 1;
            goff[g] = cd == 4 ? (H ? 36 : g == kc ? 32 : 33) * NT3 : (nb * 4 + H) * NT3 + db * T3A + da;
        }
    }

    bool flipA, flipB;
    const int Am = bc3_src(min(max(A, -1), mA + 2), mA, a.bc[2 * AXA], a.bc[2 * AXA + 1], flipA);
    const int Bm = bc3_src(min(max(B, -1), mB + 2), mB, a.bc[2 * AXB], a.bc[2 * AXB + 1], flipB);
    const long long qoffAB = (long long)(Am - 1) * a.qs[AXA] + (long long)(Bm - 1) * a.qs[AXB];
    const bool pistonB = AXB == 2 && B > mB && a.bc[5] == BC_PISTON;

    auto load_pn = [&](int pos, real& qp, real& qn) {
        bool fN;
        const int pm = bc3_src(pos, mN, a.bc[2 * AXN], a.bc[2 * AXN + 1], fN);
        const long long off = qoffAB + (long long)(pm - 1) * a.qs[AXN];
        qp = qold[off];
        qn = qold[off + CN * a.fstride];
        if (fN) qn = -qn;
        if (CN == 3) {
            const bool pist = (AXN == 2 && pos > mN && a.bc[5] == BC_PISTON) || pistonB;
            if (pist) {
                const int ci = AXN == 0 ? pos : A;
                const int cj = AXN == 1 ? pos : (AXA == 1 ? A : B);
                qn = (real)(2.0 * piston_speed(a, ci, cj, tbc)) - qn;
            }
        }
    };
    // Z and c of ring position pos, copied asynchronously
    auto load_aux = [&](int pos) {
        real* dst = saux + (pos & (RING3 - 1)) * NPL * NS3;
        const long long pofs = (long long)(pos + 1) * a.as[AXN];
        for (int e = tid; e < NS3; e += NT3P) {
            const int sa = e % S3A, sb = e / S3A;
            const int Ai = min(A0 - 2 + sa, mA + 2), Bi = min(B0 - 2 + sb, mB + 2);
            const long long o = pofs + (long long)(Ai + 1) * a.as[AXA] + (long long)(Bi + 1) * a.as[AXB];
            cp_async_el(dst + e, aux + o);
            cp_async_el(dst + NS3 + e, aux + o + a.afstride);
        }
    };
    // 1 / (Z + Z_next) along A and B of ring position pos, from its landed Z.
    // The next tile element is the next cell, or the same clamped cell past
    // the grid's last ghost.  The tile's last row and column have no next and
    // stay unset: only splits of halo slices read them, whose terms reach no
    // slice that is written.
    auto make_rcp = [&](int pos) {
        real* dst = saux + (pos & (RING3 - 1)) * NPL * NS3;
        for (int e = tid; e < NS3; e += NT3P) {
            const int sa = e % S3A, sb = e / S3A;
            if (sa == S3A - 1 || sb == S3B - 1) continue;
            const real z = dst[e];
            const real dA = z + dst[e + 1], dB = z + dst[e + S3A];
            const real rA = real(1) / dA, rB = real(1) / dB;
            // (2^-100 .. 2^100; false for NaN)
            const bool in = dA > real(7.9e-31) && dA < real(1.2e30) && dB > real(7.9e-31) && dB < real(1.2e30);
            if (!in) *far = 1;
            dst[(E1A ? 2 : 3) * NS3 + e] = rA;
            dst[(E1A ? 3 : 2) * NS3 + e] = rB;
        }
    };
    // q of this slice at position pos: role 0 stages p, role 1 the normal
    // velocity; boundary conditions are applied when the pair takes them
    auto issue_q = [&](int pos) {
        if (!active) return;
        bool fN;
        const int pm = bc3_src(pos, mN, a.bc[2 * AXN], a.bc[2 * AXN + 1], fN);
        const long long off = qoffAB + (long long)(pm - 1) * a.qs[AXN] + (H ? CN * a.fstride : 0);
        cp_async_el(sq + ((pos & 1) * 2 + H) * NT3 + sl, qold + off);
    };
    auto take_q = [&](int pos, real& qp, real& qn) {
        qp = sq[((pos & 1) * 2) * NT3 + sl];
        qn = sq[((pos & 1) * 2 + 1) * NT3 + sl];
        bool fN;
        (void)bc3_src(pos, mN, a.bc[2 * AXN], a.bc[2 * AXN + 1], fN);
        if (fN) qn = -qn;
        if (CN == 3) {
            const bool pist = (AXN == 2 && pos > mN && a.bc[5] == BC_PISTON) || pistonB;
            if (pist) {
                const int ci = AXN == 0 ? pos : A;
                const int cj = AXN == 1 ? pos : (AXA == 1 ? A : B);
                qn = (real)(2.0 * piston_speed(a, ci, cj, tbc)) - qn;
            }
        }
    };
    const int sown = (tb + 1) * S3A + (ta + 1);
    auto plane = [&](int pos, int k) -> const real* {
        return saux + (pos & (RING3 - 1)) * NPL * NS3 + k * NS3 + sown;
    };
    // split in the own direction of a fluctuation at the cell `w` across
    // (S::split with its quotients from the face reciprocals)
    bool near = true;  // the medium's sums are in range (false is sticky)
    auto split_near = [&](real xp, int pos, int w) -> Split {
        const real* Zp = plane(pos, 0);
        const real* Cp = plane(pos, 1);
        const real* Rp = plane(pos, 2 + H);  // 1 / (Z + Z_next) along the own direction
        const real zb = Zp[-OWNS + w * OTHS], zm = Zp[w * OTHS], za = Zp[OWNS + w * OTHS];
        const real b1 = -quot_rcp(xp, zb + zm, Rp[-OWNS + w * OTHS]);
        const real b2 = quot_rcp(xp, zm + za, Rp[w * OTHS]);
        const real c1 = Cp[-OWNS + w * OTHS] * b1, c2 = Cp[OWNS + w * OTHS] * b2;
        return Split{c1 * zb, -c1, c2 * za, c2};
    };
    auto split_far = [&](real xp, int pos, int w) -> Split {
        const real* Zp = plane(pos, 0);
        const real* Cp = plane(pos, 1);
        return split3_far<S>(xp, Zp[-OWNS + w * OTHS], Cp[-OWNS + w * OTHS], Zp[w * OTHS], Zp[OWNS + w * OTHS],
                             Cp[OWNS + w * OTHS]);
    };

    double cfl = 0.0;
    auto solve = [&](int i, real pL, real uL, real pR, real uR, real w[2][2], real am[2], real ap[2]) {
        real s[2];
        const real zl = *plane(i - 1, 0), cl = *plane(i - 1, 1);
        const real zr = *plane(i, 0), cr = *plane(i, 1);
        S::rpn(pL, uL, pR, uR, zl, cl, zr, cr, w, s, am, ap);
        if (i >= 1 && i <= mN + 1) {
            for (int k = 0; k < 2; ++k) {  // fmax by select: a NaN leaves cfl
                const double c = fabs(tn_d * (double)s[k]);
                cfl = c > cfl ? c : cfl;
            }
        }
    };

    load_aux(p0 - 2);
    load_aux(p0 - 1);
    load_aux(p0);
    load_aux(p0 + 1);
    issue_q(p0 + 1);
    cp_async_wait_all();
    __syncthreads();
    make_rcp(p0 - 1);
    make_rcp(p0);
    __syncthreads();
    near = *(volatile int*)far == 0;

    real wA[2][2], wB[2][2];
    real amB[2], apB[2];
    real qLp = 0, qLn = 0;
    real F0[2] = {0, 0};
    real Qs[2] = {0, 0};
    real O[2][3][2];  // own side's gadd or hadd (side, level, comp) of cell p
    for (int s_ = 0; s_ < 2; ++s_)
        for (int l = 0; l < 3; ++l)
            for (int c = 0; c < 2; ++c) O[s_][l][c] = 0;
    if (active) {
        real q0p, q0n, q1p, q1n;
        load_pn(p0 - 2, q0p, q0n);
        load_pn(p0 - 1, q1p, q1n);
        load_pn(p0, qLp, qLn);
        real am_[2], ap_[2];
        solve(p0 - 1, q0p, q0n, q1p, q1n, wA, am_, ap_);
        solve(p0, q1p, q1n, qLp, qLn, wB, amB, apB);
    }
    __syncthreads();

    const bool xch = m3 > 0 && m4 > 0;  // the pair exchanges split combinations
    // exchange planes: [side L/R][role][value] of NT3 slices each
    auto xplane = [&](int side, int role, int v) -> real* {
        return sxch + ((side * 2 + role) * 2 + v) * NT3 + sl;
    };

    for (int p = p0 - 1; p < p1; ++p) {
        const bool emit = p >= p0;
        // position p+3: its ring slot and staged q were last read before the
        // previous position's barrier
        if (p + 3 <= p1 + 1) {
            load_aux(p + 3);
            issue_q(p + 3);
        }
        near = near && *(volatile int*)far == 0;  // (set before the last barrier)
        // the reciprocals of position p+2 (its Z landed before the last barrier)
        if (p + 2 <= p1 + 1) make_rcp(p + 2);
        const real* vsrc = DIR == 0 ? qold : qnew;
        real vA = 0, vB = 0;
        // the cell values of position p+1, staged for the next position (only
        // this thread writes that cell, at that position)
        if (apply && p + 1 >= p0 && p + 1 < p1) {
            const long long off = qoffAB + (long long)p * a.qs[AXN];
            real* dv = sv + (((p + 1) & 1) * 2 + H) * 2 * NT3 + sl;
            cp_async_el(dv, vsrc + off + CA * a.fstride);
            cp_async_el(dv + NT3, vsrc + off + CB * a.fstride);
        }
        real F1[2] = {0, 0};
        real Qp[2] = {0, 0};
        real wC[2][2] = {}, amC[2] = {}, apC[2] = {}, qRp = 0, qRn = 0;
        real cq[2] = {0, 0};
        Split ma = {0, 0, 0, 0}, mp = {0, 0, 0, 0}, qm = {0, 0, 0, 0}, qp = {0, 0, 0, 0};
        const int L = p, R = p + 1;
        if (active) {
            take_q(p + 2, qRp, qRn);
            solve(p + 2, qLp, qLn, qRp, qRn, wC, amC, apC);
            real wl[2][2];
            const real sB[2] = {-*plane(p, 1), *plane(p + 1, 1)};
            for (int k = 0; k < 2; ++k) {
                wl[k][0] = wB[k][0];
                wl[k][1] = wB[k][1];
                const int lim = M::lim >= 0 ? M::lim : a.mthlim[k];
                if (order == 2 && lim > 0) {
                    const real wn2 = wB[k][0] * wB[k][0] + wB[k][1] * wB[k][1];
                    const real dl = wA[k][0] * wB[k][0] + wA[k][1] * wB[k][1];
                    const real dr = wB[k][0] * wC[k][0] + wB[k][1] * wC[k][1];
                    const real phi = phi_of<real>(lim, sB[k] > real(0) ? dl : dr, wn2);
                    wl[k][0] = phi * wB[k][0];
                    wl[k][1] = phi * wB[k][1];
                }
            }
            if (order == 2) {
                for (int k = 0; k < 2; ++k) {
                    const real as_ = fabs(sB[k]);
                    const real coef = (real(0.5) * as_) * (real(1) - as_ * dtdxave);
                    cq[0] = cq[0] + coef * wl[k][0];
                    cq[1] = cq[1] + coef * wl[k][1];
                }
            }
            F1[0] = cq[0];
            F1[1] = cq[1];
            Qp[0] = Qs[0] - tn * amB[0];
            Qp[1] = Qs[1] - tn * amB[1];
            Qs[0] = real(0) - tn * apB[0];
            Qs[1] = real(0) - tn * apB[1];

            // ---- the four rpt3 splits of interface p+1, side by side (their
            // quotients overlap): A-dq and cqxx at cell p, A+dq and cqxx at p+1
            if (m3 > 0) {
                if (near && quot_rcp_range(amB[0]) && quot_rcp_range(apB[0]) && quot_rcp_range(cq[0])) {
                    ma = split_near(amB[0], L, 0);
                    mp = split_near(apB[0], R, 0);
                    if (m3 == 2) {
                        qm = split_near(cq[0], L, 0);
                        qp = split_near(cq[0], R, 0);
                    }
                } else {
                    ma = split_far(amB[0], L, 0);
                    mp = split_far(apB[0], R, 0);
                    if (m3 == 2) {
                        qm = split_far(cq[0], L, 0);
                        qp = split_far(cq[0], R, 0);
                    }
                }
                if (m4 > 0) {
                    // the combinations the partner splits (flux3.f90:363-376, 488-495)
                    real x1 = ma.up, x3 = ma.dp, x0 = mp.up, x2 = mp.dp;
                    if (m4 == 2) {
                        x1 = ma.up + real(3) * qm.up;
                        x3 = ma.dp + real(3) * qm.dp;
                        x0 = mp.up - real(3) * qp.up;
                        x2 = mp.dp - real(3) * qp.dp;
                    }
                    *xplane(0, H, 0) = x1;
                    *xplane(0, H, 1) = x3;
                    *xplane(1, H, 0) = x0;
                    *xplane(1, H, 1) = x2;
                }
                // cell p: the amdq side of interface p+1 completes gadd/hadd
                O[0][1][0] = O[0][1][0] - H5 * ma.dp;
                O[0][1][1] = O[0][1][1] - H5 * ma.dt;
                O[1][1][0] = O[1][1][0] - H5 * ma.up;
                O[1][1][1] = O[1][1][1] - H5 * ma.ut;
            }
        }
        Split tpp = {0, 0, 0, 0}, tmp = {0, 0, 0, 0};
        if (xch) {
            pair_sync(pair_id);
            if (active) {
                const real y1 = *xplane(0, 1 - H, 0), y3 = *xplane(0, 1 - H, 1);
                const real y0 = *xplane(1, 1 - H, 0), y2 = *xplane(1, 1 - H, 1);
                Split tpm, tmm;
                if (near && quot_rcp_range(y0) && quot_rcp_range(y1) && quot_rcp_range(y2) && quot_rcp_range(y3)) {
                    tpm = split_near(y1, L, 1);
                    tmm = split_near(y3, L, -1);
                    tpp = split_near(y0, R, 1);
                    tmp = split_near(y2, R, -1);
                } else {
                    tpm = split_far(y1, L, 1);
                    tmm = split_far(y3, L, -1);
                    tpp = split_far(y0, R, 1);
                    tmp = split_far(y2, R, -1);
                }
                O[1][1][0] = O[1][1][0] + S6own * (tpm.up - tmm.up);
                O[1][1][1] = O[1][1][1] + S6own * (tpm.ut - tmm.ut);
                O[0][1][0] = O[0][1][0] + S6own * (tpm.dp - tmm.dp);
                O[0][1][1] = O[0][1][1] + S6own * (tpm.dt - tmm.dt);
                O[1][2][0] = O[1][2][0] - S6own * tpm.up;
                O[1][2][1] = O[1][2][1] - S6own * tpm.ut;
                O[0][2][0] = O[0][2][0] - S6own * tpm.dp;
                O[0][2][1] = O[0][2][1] - S6own * tpm.dt;
                O[1][0][0] = O[1][0][0] + S6own * tmm.up;
                O[1][0][1] = O[1][0][1] + S6own * tmm.ut;
                O[0][0][0] = O[0][0][0] + S6own * tmm.dp;
                O[0][0][1] = O[0][0][1] + S6own * tmm.dt;
            }
        }
        if (active) {
            if (m3 == 2) {
                O[1][1][0] = O[1][1][0] - tn * qm.up;
                O[1][1][1] = O[1][1][1] - tn * qm.ut;
                O[0][1][0] = O[0][1][0] - tn * qm.dp;
                O[0][1][1] = O[0][1][1] - tn * qm.dt;
            }
            if (emit) {
                // terms for the eight neighbours: own offset o (the side), other w (the level)
                real* out = sterm + sl;
#pragma unroll
                for (int w = -1; w <= 1; ++w)
#pragma unroll
                    for (int o = -1; o <= 1; ++o) {
                        if (o == 0 && w == 0) continue;
                        const int de1 = H ? w : o, de2 = H ? o : w;
                        const int idx9 = (de2 + 1) * 3 + (de1 + 1);
                        const int nb = idx9 < 4 ? idx9 : idx9 - 1;
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const real tv = o < 0 ? -(t_own * O[0][w + 1][c])
                                          : o == 0 ? -(t_own * (O[1][w + 1][c] - O[0][w + 1][c]))
                                                   : t_own * O[1][w + 1][c];
                            out[(nb * 4 + 2 * H + c) * NT3] = tv;
                        }
                    }
                // centre: h = 0 subtracts its own sums, te1*dG_p and te2*dH_p
                // from p and sends te1*dG_e1; h = 1 subtracts te2*dH_e2 and
                // sends te2*dH_p
                const real dp_ = t_own * (O[1][1][0] - O[0][1][0]);
                const real dv_ = t_own * (O[1][1][1] - O[0][1][1]);
                if (H == 0) {
                    out[32 * NT3] = Qp[0];
                    out[34 * NT3] = -(tn * (F1[0] - F0[0]));
                    out[33 * NT3] = -dp_;
                    out[36 * NT3] = -dv_;
                } else {
                    out[35 * NT3] = -dp_;
                    out[38 * NT3] = -dv_;
                }
            }
            // ---- cell p+1: the apdq side of interface p+1 starts gadd/hadd
            // (0 - x written as -x: the same value)
            O[0][1][0] = -(H5 * mp.dp);
            O[0][1][1] = -(H5 * mp.dt);
            O[1][1][0] = -(H5 * mp.up);
            O[1][1][1] = -(H5 * mp.ut);
            O[1][1][0] = O[1][1][0] + S6own * (tpp.up - tmp.up);
            O[1][1][1] = O[1][1][1] + S6own * (tpp.ut - tmp.ut);
            O[0][1][0] = O[0][1][0] + S6own * (tpp.dp - tmp.dp);
            O[0][1][1] = O[0][1][1] + S6own * (tpp.dt - tmp.dt);
            O[1][2][0] = -(S6own * tpp.up);
            O[1][2][1] = -(S6own * tpp.ut);
            O[0][2][0] = -(S6own * tpp.dp);
            O[0][2][1] = -(S6own * tpp.dt);
            O[1][0][0] = S6own * tmp.up;
            O[1][0][1] = S6own * tmp.ut;
            O[0][0][0] = S6own * tmp.dp;
            O[0][0][1] = S6own * tmp.dt;
            if (m3 == 2) {
                O[1][1][0] = O[1][1][0] + tn * qp.up;
                O[1][1][1] = O[1][1][1] + tn * qp.ut;
                O[0][1][0] = O[0][1][0] + tn * qp.dp;
                O[0][1][1] = O[0][1][1] + tn * qp.dt;
            }
        }
        cp_async_wait_all();
        __syncthreads();
        if (emit && apply) {
            const real* vv = sv + ((p & 1) * 2 + H) * 2 * NT3 + sl;
            vA = vv[0];
            vB = vv[NT3];
            const real* in = sterm + sl;
            if (H == 0) {
#pragma unroll
                for (int g = 0; g < NG; ++g) vA = vA + in[goff[g]] + in[goff[g] + 2 * NT3];
                vB = vB + Qp[1] - tn * (F1[1] - F0[1]);
            } else {
#pragma unroll
                for (int g = 0; g < NG; ++g) {
                    vA = vA + in[goff[g]];
                    vB = vB + in[goff[g] + 2 * NT3];
                }
            }
            const long long off = qoffAB + (long long)(p - 1) * a.qs[AXN];
            qnew[off + CA * a.fstride] = vA;
            qnew[off + CB * a.fstride] = vB;
        }
        if (active) {
            for (int k = 0; k < 2; ++k)
                for (int c = 0; c < 2; ++c) { wA[k][c] = wB[k][c]; wB[k][c] = wC[k][c]; }
            amB[0] = amC[0]; amB[1] = amC[1];
            apB[0] = apC[0]; apB[1] = apC[1];
            qLp = qRp; qLn = qRn;
            F0[0] = F1[0]; F0[1] = F1[1];
        }
        // one term buffer: every gather of p ends before a publish of p+1
        __syncthreads();
    }
    return cfl;
}

template <class S, int DIR, class M, bool LAST>
__global__ void __launch_bounds__(NT3P, CLAW_SWEEP3_MINB) sweep3p_kernel(const Sweep3Args<typename S::real> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using real = typename S::real;
    double* red = reinterpret_cast<double*>(reinterpret_cast<real*>(smem_raw) +
                                            RING3 * NPL3 * NS3 + (NTERM3 + XCH3 + QST3 + VST3) * NT3);
    __shared__ int far;  // some Z + Z' of the tile is out of quot_rcp's range for divisors
    ClawCtl* ctl = a.ctl;
    grid_dependency_sync();
    if (ctl->done) return;
    if (threadIdx.x == 0) far = 0;  // (a CTA barrier precedes the first reciprocal)
    // warps 2k (role 0) and 2k+1 (role 1) share 32 slices
    const double cfl = ((threadIdx.x >> 5) & 1) ? sweep3p_march<S, DIR, M, 1>(a, smem_raw, &far)
                                                : sweep3p_march<S, DIR, M, 0>(a, smem_raw, &far);
    if (LAST) {
        cta_cfl_and_control(ctl, cfl, red);
    } else {
        double c = cfl;
        for (int off = 16; off > 0; off >>= 1) c = fmax(c, __shfl_xor_sync(0xffffffffu, c, off));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            double m = 0.0;
            for (int w = 0; w < NT3P / 32; ++w) m = fmax(m, red[w]);
            if (!(m > 0.0)) m = (m != m) ? m : 0.0;
            atomicMax(&ctl->cfl_bits, (unsigned long long)__double_as_longlong(m));
        }
    }
}

}  // namespace clawb200
