#include "tune.h"

#include "cpsgpu_impl.h"

#include <mutex>
#include <vector>

namespace cpsgpu {

namespace {
std::mutex g_mu;
struct Entry {
  TuneKey key;
  dim3 block;
  int order;
  bool forced;  // set by the caller, not by the autotuner
};
std::vector<Entry> g_table;
}  // namespace

dim3 hop_block(const TuneKey &k, bool mix) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (auto &e : g_table)
      if (e.key == k) return e.block;
  }
  if (mix) {
    // a block holds every slice of its sites: a power of two of them, at most
    // 192 threads (FP32) or 128 (FP64, FP16, while that leaves three warps):
    // the barriers of the mixing stall one block at a time.  MatPcDagMatPc
    // with 16 / 8 sites, Mobius 24^3x64 Ls=12: FP64 5.43 / 5.46 ms, FP32
    // 2.35 / 2.45, FP16 1.84 / 1.79; 12^3x24 Ls=16: FP64 0.336 / 0.322, FP32
    // 0.182 / 0.177; 10x6x14x18 Ls=10: FP32 62 / 64 us, FP16 63 / 68
    const int ls = k.ls > 0 ? k.ls : 1;
    auto pow2 = [&](int threads) {
      int p = 1;
      while (2 * p * ls <= threads) p *= 2;
      return p;
    };
    int bx = pow2(k.prec == PREC_SINGLE ? 192 : 128);
    if (bx * ls < 96) bx = pow2(192);
    return dim3(bx, k.ls);
  }
  if (k.ls <= 1) return dim3(128, 1);
  // several slices of one 4D parity per block share their links in L1
  if (k.kind == KIND_DWF) {
    // 64 sites x 2 slices, FP64 32 x 4.  CG iteration with 64 x 2 / 32 x 4, two
    // processes each: 16^3x32 Ls=16 FP32 498, 517 / 513, 525 us, FP16 437, 439
    // / 439, 441, FP64 901, 956 / 944, 939; 12x14x20x22 Ls=12 FP32 244, 242 /
    // 254, 248, FP16 213, 211 / 217, 215, FP64 427, 430 / 411, 411
    // Other even Ls, 64 x 2 / 32 x 2 (before) / 32 x Ls/2: 16^3x32 Ls=10 FP32 327 /
    // 334 / 353, FP16 284 / 286 / 311, FP64 574 / 572 / 593, Ls=6 FP32 216 / 219 /
    // 216, FP64 358 / 361 / 366; 16^4 Ls=14 FP32 252 / 257 / 266, FP16 224 / 227 /
    // 237, FP64 407 / 403 / 440; 12^3x24 Ls=6 FP32 96 / 98 / 94
    if (k.ls % 4 == 0 && k.prec == PREC_DOUBLE) return dim3(32, 4);
    if (k.ls % 2 == 0) return dim3(64, 2);
  }
  int bs = (k.ls % 4 == 0) ? 4 : (k.ls % 2 == 0 ? 2 : 1);
  return dim3(32, bs);
}

int hop_order(const TuneKey &k) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto &e : g_table)
    if (e.key == k) return e.order;
  return ORDER_SLICES;
}

bool hop_forced(const TuneKey &k) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto &e : g_table)
    if (e.key == k) return e.forced;
  return false;
}

void tune_set(const TuneKey &k, dim3 block, int order, bool forced) {
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto &e : g_table)
    if (e.key == k) {
      e.block = block;
      e.order = order;
      e.forced = forced;
      return;
    }
  g_table.push_back({k, block, order, forced});
}

void tune_clear() {
  std::lock_guard<std::mutex> lk(g_mu);
  g_table.clear();
}

int tune_count() {
  std::lock_guard<std::mutex> lk(g_mu);
  return (int)g_table.size();
}

}  // namespace cpsgpu
