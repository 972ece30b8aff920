// FP64 complex GEMM kernels for operands whose contiguous direction is m in A and k in B.
#include <atomic>

#include "zgemm_kernel.cuh"

namespace gg {

void zgemm_launch_nk(int shape, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st) {
  zlaunch_shape<false, true, false>(shape, d, g, st);
}

}  // namespace gg
