// Instances of the tensor-core kernel: error-compensated fp16.
#include "igemm_kernel.cuh"

namespace petb200 {
PETB200_IGEMM_PICK(igemm_f16x3, kMathF16x3)
PETB200_IGEMM_WAIT_LIMIT(igemm_f16_wait_limit)
} // namespace petb200
