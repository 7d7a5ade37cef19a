// The quad-list kernels of pulse steps (every pulse of the step fixed-angle,
// applied as one rotation before the step's sums).
#include "bt_step_quad.cuh"

namespace bt {

cudaError_t launch_step_quad_rf(const StepParams<float>& p, int scheme, int vel, int prec, cudaStream_t s) {
    return launch_quad_step<false, true>(p, scheme, vel, prec, s);
}

}  // namespace bt
