// Deterministic grid reductions in FP64 and the solver's device-resident
// scalars.
//
// Every reducing kernel sums its per-thread values in a fixed order (warp
// shuffle, then warps in index order) and writes one partial per block; a
// small finalize kernel then adds one solve's partials in block order and
// updates its scalars.  Results are therefore bit-reproducible run to run,
// and the host never has to read a scalar to keep the Krylov loop going.
#pragma once
#include <cuda_runtime.h>

namespace cpsgpu {

// Solver status codes (also returned through the C ABI).
enum SolverStatus {
  ST_RUNNING = 0,
  ST_CONVERGED = 1,
  ST_MAX_ITER = 2,
  ST_BREAKDOWN = 3,  // p.Ap == 0: the reference exits the process (inv_cg.C:326-329)
  ST_NONFINITE = 4,
};

// Scalars of one Krylov solve, resident in device memory.
struct SolverScalars {
  double rr;        // |r|^2 of the iterated residual
  double rr_prev;   // previous |r|^2
  double d;         // p . A p
  double alpha, beta;
  double stop;      // stop when |r|^2 <= stop  (src_norm_sq * stop_rsd^2)
  double src_norm;  // |b|^2
  double rr_max;    // largest |r|^2 since the last reliable update
  double delta2;    // reliable-update threshold (squared)
  double shift;     // A + shift
  double sum[4];    // raw reduction results of the last finalize
  int iter;
  int max_iter;
  int done;         // SolverStatus once finished, else 0
  int reliable;     // 1 while a reliable update is pending in this iteration
  int n_reliable;   // reliable updates performed
  int pad[1];
  void *ext;        // solver-specific extension (multishift scalars)
  unsigned int pad2[4];
};

// What the finalize step does with the reduced sums.
enum ReduceOp {
  RED_STORE = 0,      // sum[] only
  RED_PAP = 1,        // sum[0] = |M p|^2, sum[1] = |p|^2: d, alpha
  RED_CG_RR = 2,      // sum[0] = |r_new|^2: iteration bookkeeping, beta
  RED_RELIABLE = 3,   // sum[0] = |b - A x|^2 (true residual): reset sloppy state
  RED_INIT = 4,       // sum[0] = |r0|^2 of the initial residual
  RED_MS_PAP = 5,     // multishift: d, b, shifted z / beta recurrences
  RED_MS_RR = 6,      // multishift: c = |r|^2, per-shift convergence
};

constexpr int MS_MAX = 64;
// iterations whose per-shift updates the multishift CG applies together
// (multishift.cu ms_flush_kernel); the loop's chunk length
constexpr int MS_DEFER = 8;

// Device-resident scalars of the multishift CG (DiracOp::MInvCG,
// minvcg.C:47-353), reached through SolverScalars::ext.
struct MsScalars {
  int nshift, iz, first, type;
  int k, max_iter, conv_all, upd_done_iter;
  double a, b, bp, c, cp, d;
  double mass[MS_MAX], rsd_sq[MS_MAX], weight[MS_MAX];
  double z[2][MS_MAX], bs[MS_MAX], as[MS_MAX];
  double rsd_out[MS_MAX];
  int conv[MS_MAX], conv_prev[MS_MAX], conv_iter[MS_MAX];
  // coefficients of the iterations since the last flush, [iteration][shift]:
  // psi_s += hf p_s where h_upd, then p_s = hz r + ha p_s where h_adv
  int nh;
  double hf[MS_DEFER][MS_MAX], hz[MS_DEFER][MS_MAX], ha[MS_DEFER][MS_MAX];
  unsigned char h_upd[MS_DEFER][MS_MAX], h_adv[MS_DEFER][MS_MAX];
};

// The shifted-system recurrences of minvcg.C: the shared scalars by thread 0
// of the finalizing block, then shift s by thread s (every thread of the
// block calls this).  One thread walking all shifts took about 1 us per
// shift (dependent loads and FP64 divisions).
__device__ inline void finalize_multishift(SolverScalars *st, int op, const double *sum) {
  MsScalars *ms = reinterpret_cast<MsScalars *>(st->ext);
  const int n = ms->nshift, s = threadIdx.x;
  __shared__ int go, any_running;
  if (op == RED_MS_PAP) {
    if (s == 0) {
      // d = <p, (A + m_0) p>   (minvcg.C:141-148, :228-236)
      const double d = sum[0] + ms->mass[0] * sum[1];
      ms->d = d;
      go = 1;
      if (!isfinite(d)) { st->done = ST_NONFINITE; go = 0; }
      else if (d == 0.0) { st->done = ST_BREAKDOWN; go = 0; }
      else {
        ms->bp = ms->b;
        ms->b = -ms->cp / d;
        ms->iz = 1 - ms->iz;
        if (ms->first) {
          ms->z[0][0] = ms->z[1][0] = 1.0;
          ms->iz = 1;
        }
        ms->bs[0] = ms->b;
        st->alpha = -ms->b;  // r += b A p is r -= alpha A p
      }
    }
    __syncthreads();
    if (!go || s == 0 || s >= n) return;
    const double b = ms->b;
    const int iz = ms->iz;
    if (ms->first) {
      // minvcg.C:152-165
      ms->z[1 - iz][s] = 1.0;
      ms->z[iz][s] = 1.0 / (1.0 - b * (ms->mass[s] - ms->mass[0]));
      ms->bs[s] = b * ms->z[iz][s];
    } else if (!ms->conv[s]) {
      // minvcg.C:238-252
      const double bp = ms->bp, a = ms->a;
      const double zt = ms->z[1 - iz][s] * ms->z[iz][s] * bp /
                        (b * a * (ms->z[iz][s] - ms->z[1 - iz][s]) +
                         ms->z[iz][s] * bp * (1 - b * (ms->mass[s] - ms->mass[0])));
      ms->bs[s] = b * zt / ms->z[1 - iz][s];
      ms->z[iz][s] = zt;
    }
    return;
  }
  // RED_MS_RR: c = |r|^2 and per-shift convergence (minvcg.C:255-304)
  const double c = sum[0];
  const bool first = ms->first;  // read by every thread before thread 0 clears it
  __syncthreads();
  if (s == 0) {
    ms->c = c;
    go = isfinite(c) ? 1 : 0;
    if (!go) st->done = ST_NONFINITE;
    any_running = 0;
    if (first) ms->first = 0;
    else if (go) ms->k += 1;
  }
  __syncthreads();
  if (!go) return;
  const int iz = ms->iz;
  const bool was = s < n && ms->conv[s];
  bool conv = was;
  if (s < n) {
    ms->conv_prev[s] = was;
    if (!first && !was) {
      const double css = c * ms->z[iz][s] * ms->z[iz][s];
      if (css < ms->rsd_sq[s]) {
        conv = true;
        ms->conv[s] = 1;
        ms->rsd_out[s] = css;
        ms->conv_iter[s] = ms->k;
      }
    }
    if (!conv) any_running = 1;
  }
  __syncthreads();
  if (s == 0) {
    ms->conv_all = first ? ((c < ms->rsd_sq[0]) ? 1 : 0) : !any_running;
    if (ms->conv_all) st->done = ST_CONVERGED;
    else if (ms->k >= ms->max_iter) st->done = ST_MAX_ITER;
    ms->a = c / ms->cp;
    ms->cp = c;
  }
  __syncthreads();
  // coefficients of this iteration's updates and of the next direction (minvcg.C:204-225)
  const int j = ms->nh;
  if (s < n) {
    const double a = ms->a;
    if (s > 0 && !conv) ms->as[s] = a * (ms->z[iz][s] * ms->bs[s]) / (ms->z[1 - iz][s] * ms->b);
    if (j < MS_DEFER) {
      ms->hf[j][s] = -ms->bs[s] * ms->weight[s];
      ms->hz[j][s] = (s == 0) ? 1.0 : ms->z[iz][s];
      ms->ha[j][s] = (s == 0) ? a : ms->as[s];
      ms->h_upd[j][s] = !was;
      ms->h_adv[j][s] = (st->done == 0) && !conv;
    }
  }
  __syncthreads();
  if (s == 0) ms->nh = j + 1;
}

__device__ __forceinline__ bool finite_d(double x) { return isfinite(x); }

__device__ inline void finalize_scalars(SolverScalars *st, int op, const double *sum) {
  for (int k = 0; k < 4; k++) st->sum[k] = sum[k];
  switch (op) {
    case RED_PAP: {
      double d = sum[0] + st->shift * sum[1];
      st->d = d;
      if (!finite_d(d)) { st->done = ST_NONFINITE; break; }
      if (d == 0.0) { st->done = ST_BREAKDOWN; break; }
      st->alpha = st->rr / d;
      break;
    }
    case RED_CG_RR: {
      double rr = sum[0];
      st->iter += 1;
      st->rr_prev = st->rr;
      st->rr = rr;
      if (!finite_d(rr)) { st->done = ST_NONFINITE; break; }
      if (st->delta2 > 0.0) {
        // mixed precision: ask for a reliable update when the iterated
        // residual has dropped by delta since the last one, or claims
        // convergence; the true residual then decides.
        if (rr > st->rr_max) st->rr_max = rr;
        if (rr <= st->stop || rr < st->delta2 * st->rr_max) {
          st->reliable = 1;
          break;
        }
      } else if (rr <= st->stop) {
        st->done = ST_CONVERGED;
        break;
      }
      if (st->iter >= st->max_iter) { st->done = ST_MAX_ITER; break; }
      st->beta = rr / st->rr_prev;
      break;
    }
    case RED_RELIABLE: {
      double rr = sum[0];
      st->n_reliable += 1;
      st->reliable = 0;
      st->rr = rr;
      st->rr_max = rr;
      if (!finite_d(rr)) { st->done = ST_NONFINITE; break; }
      if (rr <= st->stop) { st->done = ST_CONVERGED; break; }
      if (st->iter >= st->max_iter) { st->done = ST_MAX_ITER; break; }
      st->beta = rr / st->rr_prev;
      break;
    }
    case RED_INIT: {
      st->rr = sum[0];
      st->rr_max = sum[0];
      if (!finite_d(sum[0])) st->done = ST_NONFINITE;
      else if (sum[0] <= st->stop || st->max_iter <= 0) st->done = ST_CONVERGED;
      break;
    }
    default:  // RED_STORE; the multishift operations follow in finalize_multishift
      break;
  }
}

template <int NV>
__device__ __forceinline__ void warp_sum(double (&v)[NV]) {
#pragma unroll
  for (int k = 0; k < NV; k++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
}

// Global reductions are two-step and deterministic: every block of the
// reducing kernel writes its own NV partial sums (block_partial), and a
// following finalize_kernel sums one solve's partials in a fixed order and
// updates its scalars (finalize_scalars).  No block waits on another, no
// atomics: the order of the additions never depends on scheduling.

// Sum NV values over the block; thread 0 writes them as partial number blk of
// solve `solve` (partials hold NV * nblk doubles per solve).  Must be called
// by every thread of the block.
template <int NV>
__device__ void block_partial(double (&v)[NV], double *partials, unsigned solve, unsigned blk, unsigned nblk) {
  __shared__ double sm[32][NV];
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nthr = blockDim.x * blockDim.y;
  const int lane = tid & 31, warp = tid >> 5, nwarp = (nthr + 31) >> 5;
  warp_sum(v);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) sm[warp][k] = v[k];
  __syncthreads();
  if (tid == 0) {
    double *part = partials + ((size_t)solve * nblk + blk) * NV;
    for (int k = 0; k < NV; k++) {
      double s = 0.0;
      for (int w = 0; w < nwarp; w++) s += sm[w][k];
      part[k] = s;
    }
  }
}

// The common case: one solve per blockIdx.z, all its blocks in x and y.
template <int NV>
__device__ void block_partial(double (&v)[NV], double *partials) {
  block_partial<NV>(v, partials, blockIdx.z, blockIdx.x + gridDim.x * blockIdx.y, gridDim.x * gridDim.y);
}

constexpr int FINALIZE_THREADS = 1024;

// One block per solve: sum its nblk partials (thread-strided, then the warp
// and block trees, always in the same order) and finalize its scalars.  The
// gate is the one the reducing kernel had, so a solve it skipped is skipped
// here too.  The block has the warps that nblk partials fill, at most
// FINALIZE_THREADS threads (the stride, so the order of the sum does not
// depend on it): a small solve's one step from the next kernel is this
// kernel's latency.  set_cond: cond is the condition of this iteration's
// reliable update (one solve), set here instead of by a kernel of its own.
template <int NV>
__global__ void __launch_bounds__(FINALIZE_THREADS)
    finalize_kernel(const double *partials, SolverScalars *st, int op, unsigned nblk, int gate,
                    cudaGraphConditionalHandle cond = 0, int set_cond = 0) {
  const unsigned solve = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((gate == 1 && st[solve].done) ||                              // GATE_RUNNING
      (gate == 2 && (st[solve].done || !st[solve].reliable))) {     // GATE_RELIABLE
    if (tid == 0 && set_cond) cudaGraphSetConditional(cond, 0);
    return;
  }
  __shared__ double sm[FINALIZE_THREADS / 32][NV];
  const double *part = partials + (size_t)solve * nblk * NV;
  double acc[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) acc[k] = 0.0;
  // eight independent loads in flight per thread (the sum order stays fixed)
  constexpr int U = 8;
  unsigned b = tid;
  for (; b + (U - 1) * FINALIZE_THREADS < nblk; b += U * FINALIZE_THREADS) {
    double v[U][NV];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NV; k++) v[u][k] = part[(size_t)(b + u * FINALIZE_THREADS) * NV + k];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NV; k++) acc[k] += v[u][k];
  }
  for (; b < nblk; b += FINALIZE_THREADS)
#pragma unroll
    for (int k = 0; k < NV; k++) acc[k] += part[(size_t)b * NV + k];
  warp_sum(acc);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) sm[warp][k] = acc[k];
  __syncthreads();
  if (tid == 0) {
    double tot[4] = {0, 0, 0, 0};
    const int nwarp = (int)(blockDim.x >> 5);
    for (int k = 0; k < NV; k++)
      for (int w = 0; w < nwarp; w++) tot[k] += sm[w][k];
    finalize_scalars(&st[solve], op, tot);
    if (set_cond) cudaGraphSetConditional(cond, (!st[solve].done && st[solve].reliable) ? 1u : 0u);
  }
  if (op == RED_MS_PAP || op == RED_MS_RR) {
    __syncthreads();
    finalize_multishift(&st[solve], op, st[solve].sum);
  }
}

// threads of a finalize launch over nblk partials (the multishift operations
// need one per shift)
inline unsigned finalize_threads(unsigned nblk, int op) {
  unsigned t = (nblk + 31u) & ~31u;
  if ((op == RED_MS_PAP || op == RED_MS_RR) && t < (unsigned)MS_MAX) t = MS_MAX;
  return t > FINALIZE_THREADS ? FINALIZE_THREADS : t;
}

}  // namespace cpsgpu
