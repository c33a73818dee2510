// The 3D step with fused multiply-adds (CLAW_FP64_FMA) and in FP32
// (CLAW_FP32; Courant number, dt and time stay FP64), compiled with
// --fmad=true: step3f_kernel (step3d_fast.cuh) for the unsplit step, the
// split sweeps of step3ds.cuh for Godunov splitting.
#include "runner3d.cuh"
#include "step3d_fast.cuh"

namespace clawb200 {

template <typename real, int LIM, bool TRANS>
struct Step3fRunner : Runner {
    using Sh = Step3fShape<real>;
    Step3fArgs<real> args;
    int grid = 1;
    int* zrange = nullptr;  // FP32: the exponents of Z
    long long nz = 0;

    ~Step3fRunner() override {
        if (zrange) cudaFree(zrange);
    }

    int prepare(const claw_config& cfg, const Geometry& g) override {
        auto k = &step3f_kernel<real, LIM, TRANS>;
        std::memset(&args, 0, sizeof(args));
        fill_sweep3(args.g, cfg, g);
        args.tilesx = (g.mx + Sh::outx - 1) / Sh::outx;
        args.tilesy = (g.my + Sh::outy - 1) / Sh::outy;
        CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::smem));
        int dev = 0, nsm = 0, per_sm = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * Sh::rows, Sh::smem));
        if (per_sm < 1) return fail(CLAW_E_CUDA, "step3f kernel cannot be resident on an SM");
        const long long tiles = (long long)args.tilesx * args.tilesy;
        args.seglen = segment_length(tiles, g.mz, (long long)nsm * per_sm);
        const long long n = tiles * ((g.mz + args.seglen - 1) / args.seglen);
        if (n > 0x7fffffffLL) return fail(CLAW_E_UNSUPPORTED, "3D grid too large");
        grid = (int)n;
        if (sizeof(real) == 4) {
            CUDA_TRY(cudaMalloc(&zrange, 2 * sizeof(int)));
            args.zrange = zrange;
            nz = g.afstride;
        }
        return 0;
    }
    cudaError_t aux_set(cudaStream_t s) override {
        if constexpr (sizeof(real) == 4) {
            const cudaError_t e = cudaMemsetAsync(zrange, 0, 2 * sizeof(int), s);
            if (e != cudaSuccess) return e;
            impedance_range<<<(int)std::min((nz + 1023) / 1024, 592ll), 256, 0, s>>>(args.g.aux, nz, zrange);
            return cudaGetLastError();
        }
        return cudaSuccess;
    }
    cudaError_t launch(cudaStream_t s) override {
        return launch_step(&step3f_kernel<real, LIM, TRANS>, dim3(grid), dim3(32 * Sh::rows), Sh::smem, s, args);
    }
};

template <typename real>
static std::unique_ptr<Runner> step3f_runner(const claw_config& cfg) {
    if (cfg.transverse_waves < 10) return std::unique_ptr<Runner>(new Step3fRunner<real, -1, false>());
    // one limiter on both waves compiled in (128^3, us a step, FP64 / FP32: minmod 229 ->
    // 196 / 147 -> 132, superbee 234 -> 201 / 146 -> 133, van Leer 235 -> 205 / 147 -> 136,
    // MC 216 -> 202 / 147 -> 134)
    if (cfg.limiter[0] == cfg.limiter[1]) {
        const int lim = cfg.limiter[0];
        if (lim == 1) return std::unique_ptr<Runner>(new Step3fRunner<real, 1, true>());
        if (lim == 2) return std::unique_ptr<Runner>(new Step3fRunner<real, 2, true>());
        if (lim == 3) return std::unique_ptr<Runner>(new Step3fRunner<real, 3, true>());
        if (lim == 4) return std::unique_ptr<Runner>(new Step3fRunner<real, 4, true>());
    }
    return std::unique_ptr<Runner>(new Step3fRunner<real, -1, true>());
}

std::unique_ptr<Runner> make_fast_runner3d(const claw_config& cfg) {
    if (cfg.solver_id != CLAW_SOLVER_VC_ACOUSTICS_3D) return nullptr;
    if (cfg.dimensional_split > 0) {
        if (cfg.precision == CLAW_FP32)
            return std::unique_ptr<Runner>(new SplitRunner3D<VCAcoustics3D<float>, 1>());
        if (cfg.precision == CLAW_FP64_FMA)
            return std::unique_ptr<Runner>(new SplitRunner3D<VCAcoustics3D<double>, 1>());
        return nullptr;
    }
    if (cfg.precision == CLAW_FP32) return step3f_runner<float>(cfg);
    if (cfg.precision == CLAW_FP64_FMA) return step3f_runner<double>(cfg);
    return nullptr;
}

}  // namespace clawb200
