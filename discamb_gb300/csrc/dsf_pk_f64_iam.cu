// Plain-FP64 independent-atom kernels.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f64_iam(const PkArgs &A) { return dispatch_pk<double, MODEL_IAM, false, true>(A); }

}  // namespace dsf
