// Plain-FP64 Hansen-Coppens kernels, structure factors only.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f64_hc_f(const PkArgs &A) { return dispatch_pk<double, MODEL_HC, false, false>(A); }

}  // namespace dsf
