// The BF16X2 form (3 and 4 product terms).
#include "spmm_direct.cuh"

namespace dtc {

dtc_status direct_bf16x2(DirectParams& p, int W, bool four, cudaStream_t st) {
  return four ? by_block<kBF16X2, true>(p, W, st) : by_block<kBF16X2, false>(p, W, st);
}

}  // namespace dtc
