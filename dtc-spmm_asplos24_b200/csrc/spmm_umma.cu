// The tcgen05 kernels of the fp32, BF16X2 and BF16 forms.
#include "spmm_umma.cuh"

namespace dtc {

dtc_status umma_f32(DirectParams& p, int W, cudaStream_t st) {
  return umma_by_block<kF32, false>(p, W, st);
}

dtc_status umma_bf16x2(DirectParams& p, int W, bool four, cudaStream_t st) {
  return four ? umma_by_block<kBF16X2, true>(p, W, st) : umma_by_block<kBF16X2, false>(p, W, st);
}

dtc_status umma_bf16(DirectParams& p, int W, cudaStream_t st) {
  return umma_by_block<kBF16, false>(p, W, st);
}

}  // namespace dtc
