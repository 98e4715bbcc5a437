// Mixed FP32/FP64 strip step of scalar advection (fcb_step_adv.cuh): Riemann solves,
// limiter and transverse parts in FP32, flux sums, update and state in FP64.
#include "fcb_step_adv.cuh"

namespace fcb {

cudaError_t launch_step_adv_mixed(int aux_kind, int claw_version, const StepArgs& a, cudaStream_t st) {
    return launch_adv<float>(aux_kind, claw_version, a, st);
}

}  // namespace fcb
