// FP64 split step of the Euler Roe solver (fcb_step_split.cuh), compiled with
// -fmad=false so that every product and sum is rounded as in the reference.
#include "fcb_step_split.cuh"

namespace fcb {

cudaError_t launch_split_euler(int mx, int claw_version, const StepArgs& a, cudaStream_t st) {
    if (claw_version == 5) return launch_split_mx<Euler4RoeT<double, true>, 0>(mx, a, st);
    return launch_split_mx<Euler4RoeT<double, false>, 0>(mx, a, st);
}

}  // namespace fcb
