// The FP32 fast path's quad-list kernels (bt_step_quad.cuh); those of the rate
// palette and of pulse steps compile in parallel, in translation units of their
// own.
#include "bt_step_quad.cuh"

namespace bt {

cudaError_t launch_step_quad(const StepParams<float>& p, int scheme, int vel, int prec, bool pal, bool rf,
                             cudaStream_t s) {
    if (rf) return launch_step_quad_rf(p, scheme, vel, prec, s);
    if (pal) return launch_step_quad_pal(p, scheme, vel, prec, s);
    return launch_quad_step<false, false>(p, scheme, vel, prec, s);
}

}  // namespace bt
