// FP32-bulk Hansen-Coppens kernels, one atom per thread, structure factors only.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc1_f(const PkArgs &A) { return dispatch_pk<float, MODEL_HC, false, false>(A); }

}  // namespace dsf
