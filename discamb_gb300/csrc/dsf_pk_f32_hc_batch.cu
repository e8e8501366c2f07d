// Batched FP32-bulk Hansen-Coppens kernels (two atoms per thread).
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc_batch(const PkArgs &A) { return dispatch_pk_batch<F2, MODEL_HC>(A); }

}  // namespace dsf
