// Mixed FP32/FP64 split step of the systems (fcb_step_split.cuh): Riemann solves,
// limiters and transverse parts in FP32, flux sums, update and state in FP64.
#include "fcb_step_split.cuh"

namespace fcb {

cudaError_t launch_split_mixed(int solver, int mx, int claw_version, const StepArgs& a, cudaStream_t st) {
    switch (solver) {
        case SOLVER_SWE_ROE:
            if (claw_version == 5) return launch_split_mx<SweRoeT<float, true>, 0>(mx, a, st);
            return launch_split_mx<SweRoeT<float, false>, 0>(mx, a, st);
        case SOLVER_EULER4_ROE:
            if (claw_version == 5) return launch_split_mx<Euler4RoeT<float, true>, 0>(mx, a, st);
            return launch_split_mx<Euler4RoeT<float, false>, 0>(mx, a, st);
        case SOLVER_GEOCLAW_FWAVE: return launch_split_mx<GeoclawFwaveT<float>, 1>(mx, a, st);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace fcb
