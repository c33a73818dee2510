// Runners of the 3D step: the reference-order sweeps (one launch per sweep:
// x, y, z; the z-sweep's last CTA runs claw3's dt controller,
// src/3d/claw3.f:738-904) and the Godunov-split step, whose kernels the
// reference-order unit (claw3d.cu, --fmad=false) and the fused / FP32 unit
// (fast3d.cu) both build.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>

#include "host.h"
#include "riemann.cuh"
#include "step3d.cuh"
#include "step3ds.cuh"

namespace clawb200 {

// Sizes, strides, boundary conditions and method of one 3D grid.
template <typename real>
void fill_sweep3(Sweep3Args<real>& b, const claw_config& cfg, const Geometry& g) {
    std::memset(&b, 0, sizeof(b));
    b.q[0] = static_cast<real*>(g.q[0]);
    b.q[1] = static_cast<real*>(g.q[1]);
    b.aux = static_cast<const real*>(g.aux);
    b.qs[0] = 1;
    b.qs[1] = g.ld;
    b.qs[2] = g.ld * g.my;
    b.fstride = g.fstride;
    b.as[0] = 1;
    b.as[1] = g.ald;
    b.as[2] = g.ald * (g.my + 4);
    b.afstride = g.afstride;
    b.m[0] = g.mx;
    b.m[1] = g.my;
    b.m[2] = g.mz;
    for (int d = 0; d < 3; ++d) {
        b.bc[2 * d] = cfg.bc_lower[d];
        b.bc[2 * d + 1] = cfg.bc_upper[d];
    }
    b.mthlim[0] = cfg.limiter[0];
    b.mthlim[1] = cfg.limiter[1];
    b.order = cfg.order;
    b.m3 = cfg.transverse_waves / 10;
    b.m4 = cfg.transverse_waves - 10 * b.m3;
    b.d[0] = g.dx;
    b.d[1] = g.dy;
    b.d[2] = g.dz;
    b.xlower = cfg.lower[0];
    b.ylower = cfg.lower[1];
    b.ctl = g.ctl;
}

// Cells per segment of a 3D march of n cells over `tiles` tiles: the count with
// the least work in the longest column of CTAs (waves of CTAs on `slots`
// resident ones, times the cells each marches, with four cells' worth of
// start-up: halo cells and the first copies).  In 64-cell segments a 64^3 grid
// was 25 CTAs.
inline int segment_length(long long tiles, int n, long long slots) {
    long long best = -1;
    int length = n;
    for (int s = 1; s <= n; ++s) {
        const int len = (n + s - 1) / s;
        const long long ctas = tiles * ((n + len - 1) / len);
        const long long cost = (ctas + slots - 1) / slots * (len + 4);
        if (best < 0 || cost < best) {
            best = cost;
            length = len;
        }
    }
    return length;
}

// Reference order: one launch per sweep (sweep3p_kernel).
template <class S, class M>
struct Runner3D : Runner {
    using real = typename S::real;
    Sweep3Args<real> args[3];
    int grid[3] = {1, 1, 1};
    static constexpr int SMEM = sweep3_smem_bytes<real>();

    int prepare(const claw_config& cfg, const Geometry& g) override {
        const int m[3] = {g.mx, g.my, g.mz};
        int dev = 0, nsm = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        const long long slots = (long long)nsm * CLAW_SWEEP3_MINB;
        for (int dir = 0; dir < 3; ++dir) {
            const int axa = dir == 0 ? 1 : 0, axb = dir == 2 ? 1 : 2;
            fill_sweep3(args[dir], cfg, g);
            args[dir].tilesA = (m[axa] + T3A - 3) / (T3A - 2);
            args[dir].tilesB = (m[axb] + T3B - 3) / (T3B - 2);
            args[dir].seglen = segment_length((long long)args[dir].tilesA * args[dir].tilesB, m[dir], slots);
            args[dir].nseg = (m[dir] + args[dir].seglen - 1) / args[dir].seglen;
            const long long n = (long long)args[dir].tilesA * args[dir].tilesB * args[dir].nseg;
            if (n > 0x7fffffffLL) return fail(CLAW_E_UNSUPPORTED, "3D grid too large");
            grid[dir] = (int)n;
        }
        CUDA_TRY(cudaFuncSetAttribute(&sweep3p_kernel<S, 0, M, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        CUDA_TRY(cudaFuncSetAttribute(&sweep3p_kernel<S, 1, M, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        CUDA_TRY(cudaFuncSetAttribute(&sweep3p_kernel<S, 2, M, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        return 0;
    }

    cudaError_t launch(cudaStream_t s) override {
        cudaError_t e = launch_step(&sweep3p_kernel<S, 0, M, false>, dim3(grid[0]), dim3(NT3P), SMEM, s, args[0]);
        if (e == cudaSuccess) e = launch_step(&sweep3p_kernel<S, 1, M, false>, dim3(grid[1]), dim3(NT3P), SMEM, s, args[1]);
        if (e == cudaSuccess) e = launch_step(&sweep3p_kernel<S, 2, M, true>, dim3(grid[2]), dim3(NT3P), SMEM, s, args[2]);
        return e;
    }
    int launches_per_step() const override { return 3; }
};

// Godunov-split 3D step (src/3d/dimsp3.f): x-, y- and z-sweep launches over a
// scratch array of the grid plus one ghost layer.
template <class S, int BUILD>
struct SplitRunner3D : Runner {
    using real = typename S::real;
    Split3Args<real> args;
    int grid[3] = {1, 1, 1};
    real* scratch = nullptr;

    ~SplitRunner3D() override {
        if (scratch) cudaFree(scratch);
    }

    int prepare(const claw_config& cfg, const Geometry& g) override {
        std::memset(&args, 0, sizeof(args));
        for (int k = 0; k < 2; ++k) {
            args.q[k] = static_cast<const real*>(g.q[k]);
            args.qw[k] = static_cast<real*>(g.q[k]);
        }
        args.aux = static_cast<const real*>(g.aux);
        args.qs[0] = 1;
        args.qs[1] = g.ld;
        args.qs[2] = g.ld * g.my;
        args.fstride = g.fstride;
        const long long px = g.mx + 2, py = g.my + 2, pz = g.mz + 2;
        args.ps[0] = 1;
        args.ps[1] = px;
        args.ps[2] = px * py;
        args.pfstride = px * py * pz;
        args.as[0] = 1;
        args.as[1] = g.ald;
        args.as[2] = g.ald * (g.my + 4);
        args.afstride = g.afstride;
        args.m[0] = g.mx;
        args.m[1] = g.my;
        args.m[2] = g.mz;
        for (int d = 0; d < 3; ++d) {
            args.bc[2 * d] = cfg.bc_lower[d];
            args.bc[2 * d + 1] = cfg.bc_upper[d];
        }
        args.mthlim[0] = cfg.limiter[0];
        args.mthlim[1] = cfg.limiter[1];
        args.order = cfg.order;
        args.d[0] = g.dx;
        args.d[1] = g.dy;
        args.d[2] = g.dz;
        args.xlower = cfg.lower[0];
        args.ylower = cfg.lower[1];
        args.nstripx = (g.mx + DS3_STRIPX - 1) / DS3_STRIPX;
        args.nstrip32 = (int)((px + 31) / 32);
        args.ctl = g.ctl;
        // P: the four fields after the x-sweep; P2: p and v after the y-sweep
        CUDA_TRY(cudaMalloc(&scratch, (size_t)args.pfstride * 6 * sizeof(real)));
        args.P = scratch;
        args.P2 = scratch + (size_t)args.pfstride * 4;
        for (int d = 0; d < 3; ++d) args.nchunk[d] = (args.m[d] + DS3_CHUNK - 1) / DS3_CHUNK;
        int dev = 0, nsm = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        const long long ux = (long long)args.nstripx * py * pz;
        const long long uy = (long long)args.nstrip32 * pz * args.nchunk[1];
        const long long uz = (long long)args.nstrip32 * py * args.nchunk[2];
        auto ctas = [&](long long units, long long cap) {
            return (int)std::max(1LL, std::min(cap, (units + DS3_WARPS - 1) / DS3_WARPS));
        };
        grid[0] = ctas(ux, (long long)nsm * 8);
        grid[1] = ctas(uy, 1LL << 30);
        grid[2] = ctas(uz, 1LL << 30);
        return 0;
    }

    cudaError_t launch(cudaStream_t s) override {
        cudaError_t e = launch_step(split3_x_kernel<S, BUILD>, dim3(grid[0]), dim3(32 * DS3_WARPS), 0, s, args);
        if (e == cudaSuccess) e = launch_step(split3_yz_kernel<S, 1, BUILD>, dim3(grid[1]), dim3(32 * DS3_WARPS), 0, s, args);
        if (e == cudaSuccess) e = launch_step(split3_yz_kernel<S, 2, BUILD>, dim3(grid[2]), dim3(32 * DS3_WARPS), 0, s, args);
        if (e != cudaSuccess) return e;
        return cudaGetLastError();
    }
    int launches_per_step() const override { return 3; }
};

}  // namespace clawb200
