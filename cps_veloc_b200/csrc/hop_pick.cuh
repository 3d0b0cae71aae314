// The hop kernel of one (link form, epilogue, precisions, dagger) at hop
// precision P: one translation unit per precision instantiates it
// (hop_double.cu, hop_single.cu, hop_half.cu), so they compile in parallel.
#pragma once
#include "cpsgpu_impl.h"
#include "hop.cuh"

namespace cpsgpu {

using HopFn = void (*)(const HopParams, const HopViews, SolverScalars *, double *);

struct HopSel {
  int recon, ep, pr, px;
  bool dag;
  int ns;     // slices per thread (2: DWF slice pairs)
  bool halo;  // the t-slab decomposition's hop
  bool split; // four threads per site (small lattices)
};

HopFn pick_hop_double(const HopSel &q);
HopFn pick_hop_single(const HopSel &q);
HopFn pick_hop_half(const HopSel &q);

template <int P, int RECON, int EP, int PR, int PX>
HopFn get_hop(const HopSel &q) {
  if constexpr (!ep_mix(EP)) {
    if (q.split) return q.dag ? hop_split_kernel<P, RECON, EP, PR, PX, true> : hop_split_kernel<P, RECON, EP, PR, PX, false>;
  }
  // FP32 arithmetic only: the FP64 pair kernel spills kilobytes
  if constexpr (!ep_mix(EP) && P != PREC_DOUBLE) {
    if (q.ns == 2)
      return q.dag ? hop_kernel<P, RECON, EP, PR, PX, true, false, 2> : hop_kernel<P, RECON, EP, PR, PX, false, false, 2>;
  }
  return q.dag ? hop_kernel<P, RECON, EP, PR, PX, true> : hop_kernel<P, RECON, EP, PR, PX, false>;
}

template <int P, int RECON>
HopFn pick_hop_ep(const HopSel &q) {
  constexpr int PXS = (P == PREC_DOUBLE) ? PREC_DOUBLE : PREC_SINGLE;
  // the t-slab decomposition's hops: store epilogue, FP64 / FP32, 12- or 18-real links
  if (q.halo) {
    if constexpr (P != PREC_HALF) {
      if (q.ep == EP_STORE)
        return q.dag ? hop_kernel<P, RECON, EP_STORE, P, P, true, true> : hop_kernel<P, RECON, EP_STORE, P, P, false, true>;
    }
    throw Error(-2, "decomposed hop: store epilogue, FP64 or FP32");
  }
  switch (q.ep) {
    case EP_STORE: return get_hop<P, RECON, EP_STORE, P, P>(q);
    case EP_AXPY: return get_hop<P, RECON, EP_AXPY, P, P>(q);
    case EP_MIX: return get_hop<P, RECON, EP_MIX, P, P>(q);
    case EP_MIX_AXPY: return get_hop<P, RECON, EP_MIX_AXPY, P, P>(q);
    case EP_CG:
      if (q.pr == P && q.px == PXS) return get_hop<P, RECON, EP_CG, P, PXS>(q);
      break;
    case EP_MIX_CG:
      if (q.pr == P && q.px == PXS) return get_hop<P, RECON, EP_MIX_CG, P, PXS>(q);
      break;
    case EP_RES:
    case EP_MIX_RES:
      if constexpr (P == PREC_DOUBLE) {
        if (q.ep == EP_RES) {
          if (q.pr == PREC_DOUBLE) return get_hop<P, RECON, EP_RES, PREC_DOUBLE, P>(q);
          if (q.pr == PREC_SINGLE) return get_hop<P, RECON, EP_RES, PREC_SINGLE, P>(q);
          if (q.pr == PREC_HALF) return get_hop<P, RECON, EP_RES, PREC_HALF, P>(q);
        } else {
          if (q.pr == PREC_DOUBLE) return get_hop<P, RECON, EP_MIX_RES, PREC_DOUBLE, P>(q);
          if (q.pr == PREC_SINGLE) return get_hop<P, RECON, EP_MIX_RES, PREC_SINGLE, P>(q);
          if (q.pr == PREC_HALF) return get_hop<P, RECON, EP_MIX_RES, PREC_HALF, P>(q);
        }
      }
      break;
  }
  throw Error(-2, "hop: unsupported epilogue/precision combination");
}

}  // namespace cpsgpu
