// Instances of the tensor-core kernel: error-compensated TF32.
#include "igemm_kernel.cuh"

namespace petb200 {
PETB200_IGEMM_PICK(igemm_tf32x3, kMathTf32x3)
PETB200_IGEMM_WAIT_LIMIT(igemm_tf32_wait_limit)
} // namespace petb200
