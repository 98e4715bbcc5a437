// FP64 split step of the shallow-water Roe solver and the GeoClaw f-wave solver
// (fcb_step_split.cuh), compiled with -fmad=false so that every product and sum is
// rounded as in the reference.
#include "fcb_step_split.cuh"

namespace fcb {

cudaError_t launch_split_swe(int mx, int claw_version, const StepArgs& a, cudaStream_t st) {
    if (claw_version == 5) return launch_split_mx<SweRoeT<double, true>, 0>(mx, a, st);
    return launch_split_mx<SweRoeT<double, false>, 0>(mx, a, st);
}

cudaError_t launch_split_geoclaw(int mx, const StepArgs& a, cudaStream_t st) {
    return launch_split_mx<GeoclawFwaveT<double>, 1>(mx, a, st);
}

}  // namespace fcb
