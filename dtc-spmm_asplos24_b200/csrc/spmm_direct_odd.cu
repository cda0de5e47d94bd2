// The fp32 form at widths that are no multiple of 4.
#include "spmm_direct.cuh"

namespace dtc {

dtc_status direct_f32_odd(DirectParams& p, int W, cudaStream_t st) {
  return by_block<kF32Odd, false>(p, W, st);
}

}  // namespace dtc
