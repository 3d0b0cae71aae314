// Hop kernels at FP16 storage (hop_pick.cuh).
#include "hop_pick.cuh"

namespace cpsgpu {

HopFn pick_hop_half(const HopSel &q) {
  switch (q.recon) {
    case LINK_F32_18: return pick_hop_ep<PREC_HALF, LINK_F32_18>(q);
    case LINK_F32_12: return pick_hop_ep<PREC_HALF, LINK_F32_12>(q);
    case 18: return pick_hop_ep<PREC_HALF, 18>(q);
    default: return pick_hop_ep<PREC_HALF, 12>(q);
  }
}

}  // namespace cpsgpu
