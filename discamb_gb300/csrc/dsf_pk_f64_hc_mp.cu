// Plain-FP64 Hansen-Coppens kernels with the multipole adjoint.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f64_hc_mp(const PkArgs &A) { return dispatch_pk<double, MODEL_HC, true, true>(A); }

}  // namespace dsf
