// Launch configuration and template dispatch of the hop kernel (hop.cuh).
#include <algorithm>
#include <cstring>

#include "cpsgpu_impl.h"
#include "hop_pick.cuh"
#include "tune.h"

namespace cpsgpu {

namespace {

HopFn pick(int prec, const HopSel &q) {
  if (q.halo && q.recon != 12 && q.recon != 18) throw Error(-2, "decomposed hop: 12- or 18-real links");
  return prec == PREC_DOUBLE ? pick_hop_double(q) : prec == PREC_SINGLE ? pick_hop_single(q) : pick_hop_half(q);
}

// At most this many 5D sites at work on the GPU (right-hand sides and the
// other solves of a batch included) run four threads per site
// (hop_split_kernel).  Microseconds per CG iteration without / with, by sites:
// FP64 256 (Wilson 4^3x8) 37.2 / 24.7, 4096 (8^3x16) 41.2 / 31.7, 8192 (DWF
// 8^3x4 Ls=8) 44.2 / 34.2, and with the kernel forced 16384 (8^4 Ls=8) 46.7 /
// 48.9, 32768 52.7 / 64.7; FP32 inner solve 256 37.9 / 32.0, 4096 41.5 / 36.4,
// 16384 41.9 / 38.3, forced 32768 45.1 / 49.1; FP16 inner solve 256 38.9 /
// 32.8, 4096 43.1 / 39.4, 8192 45.3 / 42.1, 16384 43.2 / 40.4; 8 right-hand
// sides of 2048 sites FP64 46.8 / 48.6, FP32 48.6 / 40.5.  A batch of 4 solves
// of 16384 sites and 4 of 32768, FP32 inner: 12.8 ms, with the four threads in
// the smaller ones 14.9
constexpr long split_sites(int prec) { return prec == PREC_DOUBLE ? 8192 : 16384; }

size_t real_size(int prec) { return prec == PREC_DOUBLE ? 8 : 4; }

}  // namespace

bool hop_is_split(const Dirac &D, int prec, int nrhs, long beside) {
  return D.lat->t_nodes == 1 && D.lat->vh * D.ls * nrhs + beside <= split_sites(prec);
}

void launch_hop(const Dirac &D, const HopLaunch &L, const SpinorView &in, const SpinorView &out,
                const SpinorView &x, const SpinorView &r, const SpinorView &sol, const SpinorView &p,
                const SpinorView &b, SolverScalars *st) {
  const Lattice &lat = *D.lat;
  HopParams hp;
  memset(&hp, 0, sizeof(hp));
  for (int k = 0; k < 4; k++) {
    hp.L[k] = lat.L[k];
    hp.bc[k] = lat.bc[k];
  }
  hp.hx = lat.L[0] / 2;
  hp.dhx.init(hp.hx);
  hp.dly.init(lat.L[1]);
  hp.dlz.init(lat.L[2]);
  hp.vh = lat.vh;
  hp.ls = D.ls;
  hp.cb = L.cb;
  hp.dag = L.dag;
  hp.dwf = (D.kind == KIND_DWF);
  hp.h5 = 2.0 * D.a5inv;              // 2 / a5 (dwf_dslash_5_plus_omp.C:137)
  hp.h5wall = -2.0 * D.mass * D.a5inv; // -2 m_f / a5 (:138)
  for (int s = 0; s < D.ls && s < MAX_LS; s++) hp.coef[s] = L.coef.empty() ? 0.0 : L.coef[(size_t)s < L.coef.size() ? s : 0];
  hp.mix = L.mix;
  hp.mix_cplx = (L.mix != nullptr && D.cplx) ? 1 : 0;
  const MixScan *scan = L.mix ? D.scan_of(L.mix) : nullptr;
  if (scan) {
    hp.scan = scan->kind;
    for (int c = 0; c < 2; c++) {
      const double v[4] = {scan->rho[c], scan->w[c], scan->d[c], scan->e[c]};
      hp.scan_down[c] = scan->down[c];
      for (int k = 0; k < 4; k++) {
        hp.scan_d[c][k] = v[k];
        hp.scan_f[c][k] = (float)v[k];
      }
    }
  }
  hp.rev = lat.turn();
  hp.norm = L.norm;
  hp.red_op = L.red_op;
  hp.gate = L.gate;
  hp.face = (int)(lat.vh / lat.L[3]);
  hp.tb_fwd = (lat.t_coor == lat.t_nodes - 1) ? 1 : 0;
  hp.tb_bwd = (lat.t_coor == 0) ? 1 : 0;
  const bool split = (lat.t_nodes > 1);
  if (!split && L.sub != SUB_ALL) throw Error(-4, "interior / boundary hops: a t-partitioned lattice");
  // the interior of a slab reads no halo: the undecomposed kernel serves it
  const bool halo = split && L.sub != SUB_INTERIOR;
  if (halo && (!L.halo_fwd || !L.halo_bwd))
    throw Error(-1, "t-partitioned lattice: only the decomposed dslash (with its halos) applies the operator");
  if (split && (L.ep != EP_STORE || (L.prec != PREC_DOUBLE && L.prec != PREC_SINGLE)))
    throw Error(-2, "decomposed hop: store epilogue, FP64 or FP32");
  hp.sub = L.sub;

  HopViews v;
  v.U = lat.gauge(L.prec);
  v.in = in;
  v.out = out;
  v.x = x;
  v.r = r;
  v.sol = sol;
  v.p = p;
  v.b = b;
  v.hf = L.halo_fwd;
  v.hb = L.halo_bwd;

  const int recon = lat.recon(L.prec);
  const bool mix = ep_mix(L.ep);
  TuneKey key{L.prec, recon, L.ep, D.kind, D.ls};
  dim3 block = hop_block(key, mix);
  // block.z of a tuned shape: slices per thread (2: DWF slice pairs)
  const int ns = (block.z == 2 && hp.dwf && !mix && !halo && L.prec != PREC_DOUBLE && D.ls % (4 * (int)block.y) == 0) ? 2 : 1;
  block.z = 1;
  const bool split_mu = !mix && hop_is_split(D, L.prec, in.nrhs, L.beside) && !hop_forced(key);
  if (split_mu) block = dim3(SPLIT_BX, 1, 4);
  HopFn fn = pick(L.prec, HopSel{recon, L.ep, L.pr, L.px, L.dag != 0, ns, halo, split_mu});
  unsigned nsb;
  if (L.sub == SUB_BOUNDARY) {
    hp.subn = (hp.face + (int)block.x - 1) / (int)block.x;
    nsb = 2u * (unsigned)hp.subn;
    hp.i0 = 0;
    hp.iend = hp.face;
    hp.jump = (int)lat.vh - hp.face - hp.subn * (int)block.x;
  } else {
    const long nsites = (L.sub == SUB_INTERIOR) ? lat.vh - 2L * hp.face : lat.vh;
    if (nsites <= 0) return;  // a slab of two t-slices has no interior
    nsb = (unsigned)((nsites + block.x - 1) / block.x);
    hp.i0 = (L.sub == SUB_INTERIOR) ? hp.face : 0;
    hp.iend = hp.i0 + (int)nsites;
  }
  hp.nsg = (ns == 2 && !split_mu) ? D.ls / (2 * (int)block.y) : (D.ls + block.y - 1) / block.y;
  // ORDER_SITES: the slice groups on the grid's y (blocks run x fastest)
  const bool sites_first = (hop_order(key) == ORDER_SITES && hp.nsg > 1 && !split_mu);
  hp.spar = (hp.dwf && !mix && block.y > 1 && D.ls % (2 * block.y) == 0) ? 1 : 0;
  hp.nrhs = in.nrhs;
  hp.rtile = std::max(1, std::min(D.rhs_tile(L.prec, in.nrhs), in.nrhs));
  const unsigned ntile = (unsigned)((in.nrhs + hp.rtile - 1) / hp.rtile);
  dim3 grid = sites_first ? dim3(nsb * hp.rtile, hp.nsg, ntile) : dim3(nsb * hp.nsg * hp.rtile, 1, ntile);
  size_t smem = 0;
  if (mix) {
    smem = (size_t)D.ls * block.x * 24 * real_size(L.prec);
    if (!hp.scan) smem += 2 * (size_t)D.ls * D.ls * sizeof(double) * (D.cplx ? 2 : 1);
    // the attribute belongs to the kernel on one device: raised once per (device, kernel, size)
    struct Raised {
      int dev;
      HopFn fn;
      size_t smem;
    };
    static thread_local std::vector<Raised> raised;
    bool done = false;
    for (auto &e : raised)
      if (e.dev == lat.device && e.fn == fn && e.smem >= smem) done = true;
    if (!done) {
      CPSGPU_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      raised.push_back({lat.device, fn, smem});
    }
  }
  double *part = L.partials ? L.partials : lat.partials.as<double>();
  fn<<<grid, block, smem, lat.stream>>>(hp, v, st, part);
  CPSGPU_CUDA(cudaGetLastError());
  launch_counter()++;
  // the epilogue's reduction: per-block partials, summed and applied here
  const int nv = (ep_axpy(L.ep) && L.norm) ? 2 : (ep_cg(L.ep) || ep_res(L.ep)) ? 1 : 0;
  if (nv && st) launch_finalize(lat.stream, nv, part, st, L.red_op, nsb * hp.nsg, in.nrhs, L.gate, L.cond);
}

}  // namespace cpsgpu
