// FP32-bulk Hansen-Coppens kernels (two atoms per thread) with the position, ADP and occupancy derivatives.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_hc(const PkArgs &A) { return dispatch_pk<F2, MODEL_HC, false, true>(A); }

}  // namespace dsf
