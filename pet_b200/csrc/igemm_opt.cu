// Instances of the tensor-core kernel: the arithmetics a caller asks for by name, one TF32 product and error-compensated bf16.
#include "igemm_kernel.cuh"

namespace petb200 {
PETB200_IGEMM_PICK(igemm_tf32x1, kMathTf32x1)
PETB200_IGEMM_PICK(igemm_bf16x3, kMathBf16x3)
PETB200_IGEMM_WAIT_LIMIT(igemm_opt_wait_limit)
} // namespace petb200
