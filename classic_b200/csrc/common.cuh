// Shared device-side pieces of the wave-propagation kernels: the device
// control block (time/dt/CFL state of the claw2-style time loop), mbarrier and
// TMA helpers written directly in PTX for sm_100a, and the wave limiter.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace clawb200 {

// ----------------------------------------------------------- control block ---
// Device-resident state of one claw2-style advance (src/2d/claw2.f:494-784).
// Every step kernel reads dt / cur at entry; the last CTA to finish a step
// folds the CFL maximum and runs the accept/reject + next-dt logic here, so a
// whole time loop runs without a host round trip per step.
struct alignas(128) ClawCtl {
    // first line: read by every warp at a step's start (step_head: the first
    // 32 bytes), written by the controller alone
    double dt;
    unsigned long long wait_ns;    // limit of a device-side wait (0: the 2 s default)
    int done;
    int cur;                       // index of the buffer holding the current q
    int mode;                      // CTL_ADVANCE or CTL_SINGLE
    int skip_row;                  // test hook: 1 + the row whose copy strip 0 skips (0: none)
    double t, told, tstart, tend;
    double dt_max, cfl_max, cfl_desired;
    double cflmax_seen, dtmin, dtmax, cfl_last;
    int info, dt_variable;
    // second line: what the CTAs of a step publish
    alignas(128) unsigned long long cfl_bits;  // atomicMax target (bit pattern of a double >= 0)
    unsigned long long cfl_sweep[2];  // dimensional splitting: Courant maxima of the
                                      // y-sweep and of Strang's last x-sweep
    unsigned int ctas_done;        // last-CTA counter, reset by the last CTA
    int err;                       // device error flags (CTL_ERR_*)
    int n, maxn, nrej;             // accepted steps, step limit, rejected steps
};
static_assert(sizeof(ClawCtl) == 256, "two lines");

constexpr unsigned long long WAIT_NS_DEFAULT = 2000000000ull;

enum { CTL_ADVANCE = 0, CTL_SINGLE = 1 };

// Boundary-condition codes (mthbc in claw.data).
enum { BC_USER = 0, BC_EXTRAP = 1, BC_PERIODIC = 2, BC_WALL = 3 };
enum { CTL_ERR_TMA_TIMEOUT = 1, CTL_ERR_NAN_CFL = 2 };

// What a step kernel reads of the control block at its start: two 16-byte loads
// a warp, in flight together.  (Testing `done` before loading the rest took two
// or three L2 round trips of 0.35 us, and the block's line serves every warp of
// the grid, so its loads are few and its atomics lie elsewhere.)
struct StepHead {
    int done, cur, mode, skip_row;
    double dt;
    unsigned long long wait_ns;
};
__device__ __forceinline__ StepHead step_head(const ClawCtl* c) {
    unsigned long long d, w;
    StepHead h;
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(d), "=l"(w) : "l"(c) : "memory");
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(h.done), "=r"(h.cur), "=r"(h.mode), "=r"(h.skip_row)
                 : "l"(&c->done)
                 : "memory");
    h.dt = __longlong_as_double((long long)d);
    h.wait_ns = w ? w : WAIT_NS_DEFAULT;
    return h;
}

// The controller's operands, loaded together by the last CTA beside the Courant
// number.
struct CtlIn {
    double told, dt, tend, tstart, dt_max, cfl_max, cfl_desired, cflmax_seen, dtmin, dtmax;
    int mode, dt_variable, cur, n, maxn, nrej;
};
__device__ __forceinline__ CtlIn ctl_in(const ClawCtl* c) {
    const volatile ClawCtl* v = c;
    return CtlIn{v->told, v->dt, v->tend, v->tstart, v->dt_max, v->cfl_max, v->cfl_desired, v->cflmax_seen,
                 v->dtmin, v->dtmax, v->mode, v->dt_variable, v->cur, v->n, v->maxn, v->nrej};
}

// Controller step: identical decisions to claw2's main loop.  Runs in exactly
// one thread after every CTA of the step has published its Courant maximum
// (cfl; its slot is the caller's to clear) and its error flag (err).  The next
// launch sees the block when this grid is complete.  `stop` is what done becomes
// when the call ends (the batch kernel's mark of the launch).
__device__ __forceinline__ void ctl_finish_step(ClawCtl* c, const CtlIn& s, double cfl, int err, int stop = 1) {
    c->ctas_done = 0u;
    c->cfl_last = cfl;
    if (err) {  // a device wait gave up: the step's output is incomplete
        c->done = stop;
        return;
    }
    if (s.mode == CTL_SINGLE) {
        c->cur = s.cur ^ 1;
        return;
    }
    if (cfl != cfl) {  // NaN: stop instead of retrying forever
        c->err = err | CTL_ERR_NAN_CFL;
        c->done = stop;
        return;
    }
    const double t = s.told + s.dt;
    double dt = s.dt;
    if (cfl <= s.cfl_max) {
        c->t = t;
        c->cflmax_seen = fmax(cfl, s.cflmax_seen);
        c->cur = s.cur ^ 1;
        if (s.dt_variable) {
            if (cfl == 0.0) dt = s.dt_max;
            else dt = fmin(s.dt_max, s.dt * s.cfl_desired / cfl);
            c->dtmin = fmin(dt, s.dtmin);
            c->dtmax = fmax(dt, s.dtmax);
        }
        c->n = s.n + 1;
        if (t >= s.tend || s.n + 1 >= s.maxn) {
            c->done = stop;
        } else {
            c->told = t;
            if (t + dt > s.tend && s.tstart < s.tend) dt = s.tend - t;
        }
        c->dt = dt;
    } else {
        c->t = s.told;
        c->nrej = s.nrej + 1;
        if (s.dt_variable) {
            c->dt = fmin(s.dt_max, s.dt * s.cfl_desired / cfl);
        } else {
            c->cflmax_seen = fmax(cfl, s.cflmax_seen);
            c->done = stop;
        }
    }
}

// The step's folded Courant maximum, its slot cleared for the next step.
__device__ __forceinline__ double take_cfl(unsigned long long* slot) {
    return __longlong_as_double((long long)atomicExch(slot, 0ull));
}

// Publish one CTA's CFL maximum and, in the last CTA, run the controller.
// Call with all threads of the CTA; red must hold >= blockDim/32 doubles.
__device__ __forceinline__ void cta_cfl_and_control(ClawCtl* ctl, double cfl, double* red) {
    for (int off = 16; off > 0; off >>= 1) cfl = fmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, off));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = cfl;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
        if (!(m > 0.0)) m = (m != m) ? m : 0.0;  // canonical +0, keep NaN
        atomicMax(&ctl->cfl_bits, (unsigned long long)__double_as_longlong(m));
        __threadfence();
        const unsigned prev = atomicAdd(&ctl->ctas_done, 1u);
        if (prev == gridDim.x - 1) {
            __threadfence();
            const CtlIn in = ctl_in(ctl);
            const int err = *(volatile int*)&ctl->err;
            ctl_finish_step(ctl, in, take_cfl(&ctl->cfl_bits), err);
        }
    }
}

// The same for a step whose Courant number every CTA knows (constant speeds):
// nothing is folded, so a CTA only counts itself in.  A fence there waits for
// the CTA's last stores of q, at the end of every step; the count needs none
// unless a device wait gave up, whose flag it then orders.  Contracted FP64, us
// a step: 64^2 8.3 -> 6.4, 1024^2 18.4 -> 16.8, 4096^2 165.7 -> 160.6.
template <class F>
__device__ __forceinline__ void cta_count_and_control(ClawCtl* ctl, bool failed, F cfl_of) {
    const int any = __syncthreads_or(failed);
    if (threadIdx.x == 0) {
        if (any) __threadfence();
        unsigned prev;
        asm volatile("atom.acquire.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(&ctl->ctas_done) : "memory");
        if (prev == gridDim.x - 1) {
            const CtlIn in = ctl_in(ctl);
            const int err = *(volatile int*)&ctl->err;
            ctl_finish_step(ctl, in, cfl_of(in), err);
        }
    }
}

// ----------------------------------------------------------- PTX helpers ---
// Programmatic dependent launch: a step kernel launched with the programmatic
// stream-serialization attribute may be scheduled while the previous step's
// grid drains; it waits here, before its first read of the control block or
// q, for that grid to complete and its memory to be visible, then lets the
// next step's grid be scheduled in turn.  (Launched without the attribute,
// both instructions return at once.)  At 1024^2 the per-step time falls by
// 6-8 %: the launch and the CTAs' start-up overlap the previous grid's tail.
#ifndef CLAW_PDL
#define CLAW_PDL 1
#endif
__device__ __forceinline__ void grid_dependency_sync() {
#if CLAW_PDL
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_barrier_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait on an mbarrier phase: gives up after limit_ns of wall time
// (2 s unless the control block sets another limit) and reports failure
// instead of hanging the GPU.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  unsigned long long limit_ns = 2000000000ull) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0u && globaltimer_ns() - t0 > limit_ns) return false;
    }
}

// 3D tiled TMA load (no multicast): box -> shared memory, completion on bar.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            int w, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
        : "memory");
}

// ------------------------------------------------- contracted arithmetic ---
// Reciprocal and square root for the contracted (CLAW_FP64_FMA) kernels, by
// Newton-Raphson refinement of the hardware estimates (rcp.approx /
// rsqrt.approx, about 23 correct bits): each step doubles the correct bits,
// so two steps reach double precision to within about an ulp.  The
// reference-order kernels keep IEEE division and sqrt.
__device__ __forceinline__ double rcp_newton(double a) {
    // y <- y + y (1 - a y)
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double e = fma(-a, y, 1.0);
    y = fma(y, e, y);
    e = fma(-a, y, 1.0);
    y = fma(y, e, y);
    return y;
}
__device__ __forceinline__ float rcp_newton(float a) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
    const float e = fmaf(-a, y, 1.0f);
    return fmaf(y, e, y);
}
// sqrt(a): y ~ 1/sqrt(a) refined by y <- y (3 - a y^2) / 2 twice, then the
// root s = a y corrected once by s <- s + y (a - s^2) / 2 (Newton on s^2 = a).
// a = 0 gives 0 and a < 0 NaN, as sqrt does.
__device__ __forceinline__ double sqrt_newton(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    double h = 0.5 * a;
    y = y * fma(-h * y, y, 1.5);
    y = y * fma(-h * y, y, 1.5);
    const double s = a * y;
    const double r = fma(0.5 * y, fma(-s, s, a), s);
    return a == 0.0 ? a : r;
}

// a / b, the value of the IEEE quotient for every a and b (a zero's sign may
// differ), quick for a = 0: the compiler's FP64 division takes 148 cycles, but
// 462 when its numerator is zero (its general path), and a wave that is not
// there has a zero ratio.  A zero numerator's division becomes b / b, and the
// result is that zero, or NaN over 0 and NaN.  (Strang split 1501 x 1100, most
// cells at rest: 105 -> 81 us a step; radial 1024^2: 65 -> 57.)
template <typename real>
__device__ __forceinline__ real div_ieee(real a, real b) {
    const real q = (a != real(0) ? a : b) / b;
    return a != real(0) ? q : (fabs(b) > real(0) ? a : real(__longlong_as_double(0x7ff8000000000000ll)));
}

// x / d, correctly rounded, from r = RN(1/d): q = x r, then q += r (x - d q)
// twice.  The first correction leaves q within an ulp of x / d; then x - d q is
// exact and the second rounds correctly (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990,
// whose theorem asks for a correctly rounded reciprocal and no underflow).
// Five operations where a division takes its whole latency of 148 cycles.
// It holds for x that pass quot_rcp_range (zero, or |x| in 2^+-896) and d in
// 2^+-100; outside, the division.
__device__ __forceinline__ double quot_rcp(double x, double d, double r) {
    double q = x * r;
    q = fma(fma(-d, q, x), r, q);
    return fma(fma(-d, q, x), r, q);
}
__device__ __forceinline__ bool quot_rcp_range(double x) {
    const unsigned e = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return e - ((1023u - 896u) << 20) < (2u * 896u) << 20 || x == 0.0;
}

// Arithmetic policy of a kernel build: IEEE division and square root in the
// reference-order build (bit-identical to the CPU restatement), Newton
// reciprocals and roots in the contracted build.
template <bool FAST>
struct Arith {
    template <typename real>
    __device__ __forceinline__ static real rcp(real a) { return real(1) / a; }
    template <typename real>
    __device__ __forceinline__ static real div(real a, real b) { return div_ieee(a, b); }
    template <typename real>
    __device__ __forceinline__ static real root(real a) { return sqrt(a); }
};
template <>
struct Arith<true> {
    template <typename real>
    __device__ __forceinline__ static real rcp(real a) { return rcp_newton(a); }
    template <typename real>
    __device__ __forceinline__ static real div(real a, real b) { return a * rcp_newton(b); }
    __device__ __forceinline__ static double root(double a) { return sqrt_newton(a); }
    __device__ __forceinline__ static float root(float a) { return sqrtf(a); }
};

// ------------------------------------------------------------- limiter ---
// Limiter function phi(r) of src/2d/inlinelimiter.f90:71-97
// (1 minmod, 2 superbee, 3 van Leer, 4 MC, 5 Beam-Warming).  The minima and
// maxima are compare-and-selects whose operand order gives fmin / fmax's value
// for every r, NaN included (the constant operand wins); in FP64 fmin and fmax
// cost 20-25 cycles each on the chain of a step, a compare and select 14.
template <typename real>
__device__ __forceinline__ real phi_limiter(int meth, real r) {
    const real zero = real(0), one = real(1), two = real(2);
    auto lo = [](real m, real x) { return x < m ? x : m; };  // fmin(m, x), m not NaN
    auto hi = [](real m, real x) { return x > m ? x : m; };  // fmax(m, x), m not NaN
    switch (meth) {
        case 1: return hi(zero, lo(one, r));
        case 2: return hi(hi(zero, lo(one, two * r)), lo(two, r));
        case 3: return div_ieee(r + fabs(r), one + fabs(r));
        case 4: return hi(zero, lo(lo(two, (one + r) * real(0.5)), two * r));  // (1+r)/2 exactly
        case 5: return r;
        default: return one;
    }
}

// phi of a wave with ratio a / nn (its dot product with the upwind
// neighbour's wave over its own square), one for a zero wave (nn = 0).  A zero
// wave's quotient is 1 / 1, whose phi is one for every limiter, and a zero
// numerator's, which would take the division's general path, nn / nn: two
// compares and three selects around the division and phi, where div_ieee and
// both cases apart took four and six.  The reference-order kernels are bound by
// issue slots, of which three in four are not FP64 arithmetic: with upwind and
// the known Courant number below, radial 1024^2 50.5 -> 42.2 us a step, Strang
// 67.5 -> 54.2; this alone, 3D 128^3 1.66 -> 1.60 ms.
template <typename real>
__device__ __forceinline__ real phi_of(int meth, real a, real nn) {
    const bool live = nn != real(0), zero = live && a == real(0);
    const real den = live ? nn : real(1);
    const real p = phi_limiter<real>(meth, (live && !zero ? a : den) / den);
    if (meth < 1) return real(1);
    return zero ? (meth == 5 ? a : real(0)) : p;  // (NaN nn: a is NaN too)
}

// S::dir(mw), where a solver has it: the sign of wave mw's speed; 0 where only
// the speed itself tells.  The upwind neighbour of a wave.
template <class S, class = void>
struct wave_dir { __host__ __device__ static constexpr int of(int) { return 0; } };
template <class S>
struct wave_dir<S, decltype((void)S::dir(0))> { __host__ __device__ static constexpr int of(int mw) { return S::dir(mw); } };
template <class S, typename real>
__device__ __forceinline__ real upwind(int mw, real s, real left, real right) {
    const int d = wave_dir<S>::of(mw);
    if (d != 0) return d > 0 ? left : right;
    return s > real(0) ? left : right;
}

// The Courant number of a solver whose speeds are one constant (S::top_speed),
// where no capacity scales them, needs no face: every face has it.
template <class S, class = void>
struct const_speed { static constexpr bool value = false; };
template <class S>
struct const_speed<S, decltype((void)&S::top_speed)> { static constexpr bool value = true; };

// Courant number of a sweep whose faces all carry the speeds -c and c: the larger
// of dt/dx s and -dt/dx s over both is |dt/dx| c, for a backward step (dt < 0)
// too.  Zero for a NaN, which a fold over faces drops.
__device__ __forceinline__ double sweep_cfl(double dtdx, double c) {
    const double v = fabs(dtdx * c);
    return v > 0.0 ? v : 0.0;
}

// min(x, 0) and max(x, 0), fmin's and fmax's values (zero for a NaN)
template <typename real>
__device__ __forceinline__ real neg_part(real x) { return x < real(0) ? x : real(0); }
template <typename real>
__device__ __forceinline__ real pos_part(real x) { return x > real(0) ? x : real(0); }

// Fold a face's Courant number c into m (not NaN): fmax(m, c), by a select.
__device__ __forceinline__ double fold_cfl(double m, double c) { return c > m ? c : m; }

// phi(r) of the contracted build: the same functions by compare-and-select
// (no fmin/fmax, whose NaN rules cost extra FP64 instructions) and a Newton
// reciprocal in van Leer's quotient.
template <typename real>
__device__ __forceinline__ real phi_limiter_fast(int meth, real r) {
    const real zero = real(0), one = real(1), two = real(2);
    auto mn = [](real a, real b) { return a < b ? a : b; };
    auto mx = [](real a, real b) { return a > b ? a : b; };
    switch (meth) {
        case 1: return mx(zero, mn(one, r));
        case 2: return mx(mx(zero, mn(one, two * r)), mn(two, r));
        case 3: {
            const real ar = fabs(r);
            return (r + ar) * rcp_newton(one + ar);
        }
        case 4: return mx(zero, mn(mn((one + r) * real(0.5), two), two * r));
        case 5: return r;
        default: return one;
    }
}

}  // namespace clawb200
