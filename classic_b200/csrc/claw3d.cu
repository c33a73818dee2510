// The 3D step in the reference's order of operations (--fmad=false):
// bit-identical to the CPU restatement of step3 / flux3 / claw3, and of
// dimsp3 / step3ds when dimensional splitting is on.  FP32 and fused FP64 go
// to the contracted build (fast3d.cu).
#include "runner3d.cuh"

namespace clawb200 {

std::unique_ptr<Runner> make_runner3d(const claw_config& cfg) {
    if (cfg.solver_id != CLAW_SOLVER_VC_ACOUSTICS_3D) return nullptr;
    if (cfg.precision != CLAW_FP64) return make_fast_runner3d(cfg);
    // src/3d/claw3ez.f:136: any splitting request runs dimsp3's Godunov splitting
    if (cfg.dimensional_split > 0)
        return std::unique_ptr<Runner>(new SplitRunner3D<VCAcoustics3D<double>, 0>());
    using S = VCAcoustics3D<double>;
    // one limiter on both waves compiled in (128^3, us a step: minmod 1888 ->
    // 1600, superbee 1884 -> 1612, van Leer 1929 -> 1695, MC 1911 -> 1622)
    if (cfg.order == 2 && cfg.transverse_waves == 22 && cfg.limiter[0] == cfg.limiter[1]) {
        const int lim = cfg.limiter[0];
        if (lim == 1) return std::unique_ptr<Runner>(new Runner3D<S, Method3D<2, 2, 1>>());
        if (lim == 2) return std::unique_ptr<Runner>(new Runner3D<S, Method3D<2, 2, 2>>());
        if (lim == 3) return std::unique_ptr<Runner>(new Runner3D<S, Method3D<2, 2, 3>>());
        if (lim == 4) return std::unique_ptr<Runner>(new Runner3D<S, MethodMC3D>());
    }
    return std::unique_ptr<Runner>(new Runner3D<S, MethodGeneric3D>());
}

}  // namespace clawb200
