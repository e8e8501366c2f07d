// FP32-bulk independent-atom kernels (two atoms per thread), structure factors only.  2,000 atoms, 50,021 reflections:
// P2_1, isotropic 181 us, with the derivatives computed and dropped 286, sf_grad_body without the derivatives 209;
// P2_1/c, anisotropic 230, 328 and 309; 100 atoms, 3,001 reflections, P2_1/c 27, 38 and 38.
#include "dsf_pk_launch.cuh"

namespace dsf {

cudaError_t launch_pk_f32_iam_f(const PkArgs &A) { return dispatch_pk<F2, MODEL_IAM, false, false>(A); }

}  // namespace dsf
