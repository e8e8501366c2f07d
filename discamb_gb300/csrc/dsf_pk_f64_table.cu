// Plain-FP64 tabulated-form-factor kernels.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f64_table(const PkArgs &A) { return dispatch_pk<double, MODEL_TABLE, false, true>(A); }

}  // namespace dsf
