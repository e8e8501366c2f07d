// FP32-bulk Hansen-Coppens kernels (two atoms per thread), structure factors only.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc_f(const PkArgs &A) { return dispatch_pk<F2, MODEL_HC, false, false>(A); }

}  // namespace dsf
