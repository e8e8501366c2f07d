// Batched FP32-bulk Hansen-Coppens kernels, one atom per thread.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc1_batch(const PkArgs &A) { return dispatch_pk_batch<float, MODEL_HC>(A); }

}  // namespace dsf
