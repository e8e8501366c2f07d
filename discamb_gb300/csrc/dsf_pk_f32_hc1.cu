// FP32-bulk Hansen-Coppens kernels, one atom per thread (structures with a type per atom).
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc1(const PkArgs &A) { return dispatch_pk<float, MODEL_HC, false, true>(A); }

}  // namespace dsf
