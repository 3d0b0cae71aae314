// Hop kernels at FP64 (hop_pick.cuh).
#include "hop_pick.cuh"

namespace cpsgpu {

HopFn pick_hop_double(const HopSel &q) {
  return q.recon == 18 ? pick_hop_ep<PREC_DOUBLE, 18>(q) : pick_hop_ep<PREC_DOUBLE, 12>(q);
}

}  // namespace cpsgpu
