// The quad-list kernels with per-voxel rates (the rate palette).
#include "bt_step_quad.cuh"

namespace bt {

cudaError_t launch_step_quad_pal(const StepParams<float>& p, int scheme, int vel, int prec, cudaStream_t s) {
    return launch_quad_step<true, false>(p, scheme, vel, prec, s);
}

}  // namespace bt
