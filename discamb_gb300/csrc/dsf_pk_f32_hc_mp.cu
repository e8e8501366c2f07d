// FP32-bulk Hansen-Coppens kernels with the multipole adjoint.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc_mp(const PkArgs &A) { return dispatch_pk<float, MODEL_HC, true, true>(A); }

}  // namespace dsf
