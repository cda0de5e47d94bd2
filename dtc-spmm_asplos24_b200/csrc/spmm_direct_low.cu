// The BF16 and FP8 forms.
#include "spmm_direct.cuh"

namespace dtc {

dtc_status direct_bf16(DirectParams& p, int W, cudaStream_t st) {
  return by_block<kBF16, false>(p, W, st);
}

dtc_status direct_fp8(DirectParams& p, int W, cudaStream_t st) {
  return by_block<kFP8, false>(p, W, st);
}

}  // namespace dtc
