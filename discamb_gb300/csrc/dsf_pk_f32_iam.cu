// FP32-bulk independent-atom kernels (two atoms per thread).
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_iam(const PkArgs &A) { return dispatch_pk<F2, MODEL_IAM, false, true>(A); }

}  // namespace dsf
