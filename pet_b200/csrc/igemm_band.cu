// Instances of the tensor-core kernel: the banded products.
#include "igemm_kernel.cuh"

namespace petb200 {
KernelFn igemm_band(int band, int pp) {
    if (band == 1) // persistent mode with an epilogue of its own
        return k_igemm<true, kMathTf32x3, kNarrow, 1>;
    return pp == kSingle ? k_igemm<true, kMathTf32x3, kSingle, 2>
                         : (pp == kNarrow ? k_igemm<true, kMathTf32x3, kNarrow, 2> : k_igemm<true, kMathTf32x3, kWide, 2>);
}
PETB200_IGEMM_WAIT_LIMIT(igemm_band_wait_limit)
} // namespace petb200
