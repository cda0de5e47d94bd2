// The SPLIT24 form (3 and 4 product terms).
#include "spmm_direct.cuh"

namespace dtc {

dtc_status direct_split24(DirectParams& p, int W, bool four, cudaStream_t st) {
  return four ? by_block<kSplit24, true>(p, W, st) : by_block<kSplit24, false>(p, W, st);
}

}  // namespace dtc
