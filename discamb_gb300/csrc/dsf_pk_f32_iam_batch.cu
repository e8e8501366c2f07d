// Batched FP32-bulk independent-atom kernels (two atoms per thread).
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_iam_batch(const PkArgs &A) { return dispatch_pk_batch<F2, MODEL_IAM>(A); }

}  // namespace dsf
