// Plain-FP64 Hansen-Coppens kernels with the position, ADP and occupancy derivatives.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f64_hc(const PkArgs &A) { return dispatch_pk<double, MODEL_HC, false, true>(A); }

}  // namespace dsf
