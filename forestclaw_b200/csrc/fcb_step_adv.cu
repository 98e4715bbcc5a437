// FP64 strip step of scalar advection (fcb_step_adv.cuh), compiled with -fmad=false so
// that every product and sum is rounded as in the reference.
#include "fcb_step_adv.cuh"

namespace fcb {

cudaError_t launch_step_adv(int aux_kind, int claw_version, const StepArgs& a, cudaStream_t st) {
    return launch_adv<double>(aux_kind, claw_version, a, st);
}

}  // namespace fcb
