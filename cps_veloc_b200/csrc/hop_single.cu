// Hop kernels at FP32 (hop_pick.cuh).
#include "hop_pick.cuh"

namespace cpsgpu {

HopFn pick_hop_single(const HopSel &q) {
  return q.recon == 18 ? pick_hop_ep<PREC_SINGLE, 18>(q) : pick_hop_ep<PREC_SINGLE, 12>(q);
}

}  // namespace cpsgpu
