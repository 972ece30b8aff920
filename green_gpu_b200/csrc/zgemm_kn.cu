// FP64 complex GEMM kernels for operands whose contiguous direction is k in A and n in B.
#include <atomic>

#include "zgemm_kernel.cuh"

namespace gg {

void zgemm_launch_kn(int shape, bool g3, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st) {
  if (g3) zlaunch_shape<true, false, true>(shape, d, g, st);
  else zlaunch_shape<true, false, false>(shape, d, g, st);
}

}  // namespace gg
