// The Ls x Ls chirality mixing as a recurrence along s.
//
// With the same real b, c on every slice all matrices of the Mobius operator
// are functions of one shift S (slice s from s-1, the wall weighted -m, or
// its mirror image from s+1): either B = d + e S (zmobius_dslash_4's mixing,
// 1 + K D5) or a + g (1 + K S)^-1 (M5^-1, B M5^-1 and the products with
// kappa_b, their adjoints, the MIT forms).  So out = d x + e y with
//   band:  y_0 = w x_{n-1},        y_s = x_{s-1}
//   scan:  h = sum_t rho^(n-1-t) x_t (Horner),  y_0 = w h,
//          y_s = rho y_{s-1} + x_{s-1}
// (rho = -K; zmobius_m5inv.C:247-396 solves the same bidiagonal-plus-corner
// system): 4 multiply-adds per real whatever Ls is, where the dense matrix
// takes Ls.  d = a + g and e = g rho are of the size of the matrix; a and g
// alone are not (B M5^-1 has a = c / K, 21 at b = 1.5, c = 0.5, M5 = 1.8 for
// entries up to 1.5), so a sum of a x and g y would cancel.
//
// fit_mix_scan recognises the form in the packed matrices; what does not have
// it (slices with different real b_s, c_s, complex ones, |K| > 0.6, Ls < 3)
// keeps the dense kernels.  Error of one mixing in the 2-norm, of the exact
// one, dense / this, 6 <= Ls <= 32, 0.001 <= m <= 0.5: FP32 2.5e-8 - 1.5e-7 /
// 2.5e-8 - 1.1e-7, FP64 6e-17 - 2.8e-16 / 5e-17 - 1.6e-16, and matrix by
// matrix up to |K| = 0.6 at most 1.2 times the dense one's, 0.6 times in the
// mean; from 0.65 on single ones reach 1.3 times, at 0.85 2 times (rho^k
// carries k roundings of rho).
//
// FP64, FP32: a thread per 16-byte group of one site holds its Ls values in
// registers (all loads in flight at once), so each field is read and written
// once and the kernel is HBM bound.  FP16: half a warp per chirality of 16
// sites, a thread holding the 12 stored values of every slice of its site
// and the site's norms; the new norm is the larger of the two chiralities'
// maxima (shuffles).  Measured (M5^-1, 24^3x64, Ls = 12, dense
// kernel / this): FP64 467 / 330 us (6.2 TB/s), FP32 193 / 160 us
// (6.4 TB/s), FP16 174 / 110 us (5.0 TB/s); MatPcDagMatPc, with the hop's
// mixing epilogue in the same form: FP64 5.80 / 5.43 ms, FP32 2.53 / 2.26 ms,
// FP16 2.11 / 1.81 ms
#include <cmath>

#include "cpsgpu_impl.h"
#include "hop.cuh"

namespace cpsgpu {

namespace {

// coefficients of one chirality in the arithmetic precision
template <typename R> struct ScanCoef {
  R rho, w, d, e;
  int down;
};
template <typename R> struct ScanArg {
  ScanCoef<R> c[2];  // upper, lower chirality
};

__device__ __forceinline__ double2 fma2(double s, double2 x, double2 y) { return make_double2(fma(s, x.x, y.x), fma(s, x.y, y.y)); }
__device__ __forceinline__ float4 fma2(float s, float4 x, float4 y) {
  const float2 a = __ffma2_rn(make_float2(s, s), make_float2(x.x, x.y), make_float2(y.x, y.y));
  const float2 b = __ffma2_rn(make_float2(s, s), make_float2(x.z, x.w), make_float2(y.z, y.w));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ double2 mul2(double s, double2 x) { return make_double2(s * x.x, s * x.y); }
__device__ __forceinline__ float4 mul2(float s, float4 x) { return make_float4(s * x.x, s * x.y, s * x.z, s * x.w); }

constexpr int SCAN_SITES = 32;

// LS > 0: the Ls values in registers; LS = 0: any Ls, the input read twice
// (the second time from L1 / L2)
template <int P, int LS, bool BAND>
__global__ void __launch_bounds__(SCAN_SITES * PrecTraits<P>::NG)
    scan_kernel(SpinorView in, SpinorView out, const ScanArg<typename PrecTraits<P>::real> arg, int ls,
                const SolverScalars *st, int gate, int rev) {
  using R = typename PrecTraits<P>::real;
  using T = typename std::conditional<P == PREC_DOUBLE, double2, float4>::type;
  constexpr int NG = PrecTraits<P>::NG;
  if (gate == GATE_RUNNING && st[blockIdx.z].done) return;
  if (gate == GATE_RELIABLE && (st[blockIdx.z].done || !st[blockIdx.z].reliable)) return;
  const int n = LS > 0 ? LS : ls;
  const int g = threadIdx.y;
  const long i = (long)(rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * SCAN_SITES + threadIdx.x;
  if (i >= in.vh) return;
  const ScanCoef<R> c = arg.c[g >= NG / 2];  // uniform in a warp
  const long rhs = blockIdx.z, step = (c.down ? -1L : 1L) * NG * in.vh;
  const long first = ((rhs * n + (c.down ? n - 1 : 0)) * NG + g) * in.vh + i;
  const T *ip = reinterpret_cast<const T *>(in.data) + first;
  T *op = reinterpret_cast<T *>(out.data) + first;
  if constexpr (LS > 0) {
    T x[LS];
#pragma unroll
    for (int k = 0; k < LS; k++) x[k] = __ldg(ip + k * step);
    T y;
    if constexpr (BAND) {
      y = mul2(c.w, x[LS - 1]);
    } else {
      T h = x[0];
#pragma unroll
      for (int k = 1; k < LS; k++) h = fma2(c.rho, h, x[k]);
      y = mul2(c.w, h);
    }
#pragma unroll
    for (int k = 0; k < LS; k++) {
      op[k * step] = fma2(c.e, y, mul2(c.d, x[k]));
      if (k + 1 < LS) y = BAND ? x[k] : fma2(c.rho, y, x[k]);
    }
  } else {
    T y;
    const T x0 = __ldg(ip);
    if constexpr (BAND) {
      y = mul2(c.w, __ldg(ip + (n - 1) * step));
    } else {
      T h = x0;
#pragma unroll 4
      for (int k = 1; k < n; k++) h = fma2(c.rho, h, __ldg(ip + k * step));
      y = mul2(c.w, h);
    }
    T x = x0;
    for (int k = 0; k < n; k++) {
      const T xn = k + 1 < n ? __ldg(ip + (k + 1) * step) : x;
      op[k * step] = fma2(c.e, y, mul2(c.d, x));
      y = BAND ? x : fma2(c.rho, y, x);
      x = xn;
    }
  }
}

constexpr int SCAN_HALF_TPB = 128;

// FP16: the chirality's 12 values of one slice as stored (6 words) and unpacked
struct Half12 {
  uint4 q;
  uint2 e;
};
// lower = 0: reals 0-7 are group 0, 8-11 the first half of group 1; lower = 1: 12-15 its second half, 16-23 group 2
__device__ __forceinline__ void unpack12(const Half12 &v, int lower, float2 (&f)[6]) {
  // the six words in storage order
  const unsigned w[6] = {lower ? v.e.x : v.q.x, lower ? v.e.y : v.q.y, lower ? v.q.x : v.q.z,
                         lower ? v.q.y : v.q.w, lower ? v.q.z : v.e.x, lower ? v.q.w : v.e.y};
#pragma unroll
  for (int k = 0; k < 6; k++) f[k] = __half22float2(*reinterpret_cast<const __half2 *>(&w[k]));
}

// blocks per SM that the registers have to allow: at Ls = 12 two instead of
// three take 132 us instead of 109 (24^3x64), at 9 three instead of four 18.6
// instead of 16.7 (16^3x32)
template <int LS, bool BAND> constexpr int scan_half_blocks() {
  if (BAND) return LS <= 8 ? 4 : LS <= 12 ? 3 : 2;
  return LS <= 4 ? 6 : LS <= 6 ? 5 : LS <= 9 ? 4 : LS <= 12 ? 3 : 2;
}

template <int LS, bool BAND>
__global__ void __launch_bounds__(SCAN_HALF_TPB, (scan_half_blocks<LS, BAND>()))
    scan_half_kernel(SpinorView in, SpinorView out, const ScanArg<float> arg, const SolverScalars *st, int gate, int rev) {
  if (gate == GATE_RUNNING && st[blockIdx.z].done) return;
  if (gate == GATE_RELIABLE && (st[blockIdx.z].done || !st[blockIdx.z].reliable)) return;
  const int lane = threadIdx.x & 31, lower = lane >> 4;
  const int i = (rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * (SCAN_HALF_TPB / 2) + (threadIdx.x >> 5) * 16 + (lane & 15);
  const int vh = (int)in.vh;
  const bool active = i < vh;
  const ScanCoef<float> c = arg.c[lower];
  const long rhs = blockIdx.z;
  const long base = rhs * LS + (c.down ? LS - 1 : 0), dir = c.down ? -1 : 1;
  const uint4 *ip = reinterpret_cast<const uint4 *>(in.data);
  uint4 *op = reinterpret_cast<uint4 *>(out.data);
  Half12 x[LS];
  float nrm[LS];
  if (active) {
#pragma unroll
    for (int k = 0; k < LS; k++) {
      const long sl = base + dir * k;
      const uint4 *d = ip + sl * 3 * vh + i;
      x[k].q = __ldg(d + (lower ? 2 * vh : 0));
      x[k].e = __ldg(reinterpret_cast<const uint2 *>(d + vh) + lower);
      nrm[k] = __ldg(in.norm + sl * vh + i);
    }
  } else {
#pragma unroll
    for (int k = 0; k < LS; k++) {
      x[k].q = make_uint4(0, 0, 0, 0);
      x[k].e = make_uint2(0, 0);
      nrm[k] = 0.f;
    }
  }
  auto value = [&](int k, float2 (&f)[6]) {
    unpack12(x[k], lower, f);
#pragma unroll
    for (int q = 0; q < 6; q++) f[q] = __fmul2_rn(f[q], make_float2(nrm[k], nrm[k]));
  };
  const float2 rho = make_float2(c.rho, c.rho), w = make_float2(c.w, c.w), d = make_float2(c.d, c.d),
               e = make_float2(c.e, c.e);
  float2 y[6], v[6];
  if constexpr (BAND) {
    value(LS - 1, v);
#pragma unroll
    for (int q = 0; q < 6; q++) y[q] = __fmul2_rn(w, v[q]);
    value(0, v);
  } else {
    float2 h[6];
    value(0, h);
#pragma unroll
    for (int k = 1; k < LS; k++) {
      value(k, v);
#pragma unroll
      for (int q = 0; q < 6; q++) h[q] = __ffma2_rn(rho, h[q], v[q]);
    }
#pragma unroll
    for (int q = 0; q < 6; q++) y[q] = __fmul2_rn(w, h[q]);
    value(0, v);
  }
  // out = d x + e y; its norm needs the other chirality's maximum for the same
  // slice, and the two recurrences run through the slices from opposite ends:
  // at step k one is at slice k, the other at LS-1-k.  So the first half of
  // the outputs waits in registers, and step k of the second half finishes
  // its own slice and the kept one of step LS-1-k.
  auto finish = [&](int k, const float2 (&o)[6], float m) {
    const float inv = (m > 0.f) ? 1.0f / m : 0.f;
    unsigned r[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const __half2 hh = __floats2half2_rn(o[q].x * inv, o[q].y * inv);
      r[q] = *reinterpret_cast<const unsigned *>(&hh);
    }
    if (active) {
      const long sl = base + dir * k;
      uint4 *d = op + sl * 3 * vh + i;
      d[lower ? 2 * vh : 0] = lower ? make_uint4(r[2], r[3], r[4], r[5]) : make_uint4(r[0], r[1], r[2], r[3]);
      reinterpret_cast<uint2 *>(d + vh)[lower] = lower ? make_uint2(r[0], r[1]) : make_uint2(r[4], r[5]);
      if (!lower) out.norm[sl * vh + i] = m;
    }
  };
  float2 keep[LS / 2][6];
  float mk[LS / 2];
#pragma unroll
  for (int k = 0; k < LS; k++) {
    if (k > 0) value(k, v);
    float2 o[6];
    float m = 0.f;
#pragma unroll
    for (int q = 0; q < 6; q++) {
      o[q] = __ffma2_rn(e, y[q], __fmul2_rn(d, v[q]));
      m = fmaxf(m, fmaxf(fabsf(o[q].x), fabsf(o[q].y)));
    }
    if (k + 1 < LS) {
#pragma unroll
      for (int q = 0; q < 6; q++) y[q] = BAND ? v[q] : __ffma2_rn(rho, y[q], v[q]);
    }
    if (k < LS / 2) {
#pragma unroll
      for (int q = 0; q < 6; q++) keep[k][q] = o[q];
      mk[k] = m;
    } else if (2 * k + 1 == LS) {  // the middle slice of an odd Ls: both are there
      finish(k, o, fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16)));
    } else {
      const int q = LS - 1 - k;
      const float other_now = __shfl_xor_sync(0xffffffffu, m, 16), other_kept = __shfl_xor_sync(0xffffffffu, mk[q], 16);
      finish(k, o, fmaxf(m, other_kept));
      finish(q, keep[q], fmaxf(mk[q], other_now));
    }
  }
}

template <typename R> ScanArg<R> scan_arg(const MixScan &m) {
  ScanArg<R> a;
  for (int k = 0; k < 2; k++) a.c[k] = {R(m.rho[k]), R(m.w[k]), R(m.d[k]), R(m.e[k]), m.down[k]};
  return a;
}

template <int P, int LS>
void launch_full(const MixScan &m, const SpinorView &in, const SpinorView &out, int ls, const SolverScalars *st, int gate,
                 cudaStream_t s, int rev) {
  using R = typename PrecTraits<P>::real;
  const ScanArg<R> a = scan_arg<R>(m);
  const dim3 block(SCAN_SITES, PrecTraits<P>::NG);
  const dim3 grid((unsigned)((in.vh + SCAN_SITES - 1) / SCAN_SITES), 1, in.nrhs);
  if (m.kind == MixScan::BAND) scan_kernel<P, LS, true><<<grid, block, 0, s>>>(in, out, a, ls, st, gate, rev);
  else scan_kernel<P, LS, false><<<grid, block, 0, s>>>(in, out, a, ls, st, gate, rev);
}

template <int LS>
void launch_half(const MixScan &m, const SpinorView &in, const SpinorView &out, const SolverScalars *st, int gate,
                 cudaStream_t s, int rev) {
  const ScanArg<float> a = scan_arg<float>(m);
  const dim3 grid((unsigned)((in.vh + SCAN_HALF_TPB / 2 - 1) / (SCAN_HALF_TPB / 2)), 1, in.nrhs);
  if (m.kind == MixScan::BAND) scan_half_kernel<LS, true><<<grid, SCAN_HALF_TPB, 0, s>>>(in, out, a, st, gate, rev);
  else scan_half_kernel<LS, false><<<grid, SCAN_HALF_TPB, 0, s>>>(in, out, a, st, gate, rev);
}

// one chirality; m(i, j) the matrix seen from the end the recurrence starts at
template <typename F>
bool fit(int n, F &&m, double scale, MixScan &s, int c, int down, int kind) {
  const double tol = 1e-15 * scale;  // some roundings of the matrix product it came from
  const double corner = m(0, n - 1), d1 = m(1, 0);
  const double rho = kind == MixScan::BAND ? 0.0 : m(2, 0) / d1;
  if (d1 == 0.0 || !(std::fabs(rho) <= 0.6) || (kind == MixScan::SCAN && rho == 0.0)) return false;
  const double e = d1 - corner * std::pow(rho, n), w = corner / e, d = m(0, 0) - corner * std::pow(rho, n - 1);
  if (!std::isfinite(w)) return false;
  // (pow(0, 0) is 1)
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      const double model = (i == j ? d : 0.0) + e * ((i > j ? std::pow(rho, i - 1 - j) : 0.0) + w * std::pow(rho, n - 1 - j + i));
      if (!(std::fabs(m(i, j) - model) <= tol)) return false;
    }
  s.rho[c] = rho;
  s.w[c] = w;
  s.d[c] = d;
  s.e[c] = e;
  s.down[c] = down;
  return true;
}

}  // namespace

MixScan fit_mix_scan(int n, const std::vector<double> &h) {
  MixScan s;
  if (n < 3 || h.size() != 2 * (size_t)n * n) return s;
  for (int kind : {(int)MixScan::BAND, (int)MixScan::SCAN}) {
    bool ok = true;
    for (int c = 0; c < 2 && ok; c++) {
      const double *M = h.data() + (size_t)c * n * n;
      double scale = 0.0;
      for (int k = 0; k < n * n; k++) scale = std::max(scale, std::fabs(M[k]));
      ok = fit(n, [&](int i, int j) { return M[i * n + j]; }, scale, s, c, 0, kind) ||
           fit(n, [&](int i, int j) { return M[(n - 1 - i) * n + (n - 1 - j)]; }, scale, s, c, 1, kind);
    }
    if (ok && s.down[0] != s.down[1]) {  // the two chiralities mirror each other
      s.kind = kind;
      return s;
    }
  }
  return MixScan();
}

bool launch_mix_scan(const Dirac &D, int prec, const double *mix, const SpinorView &in, const SpinorView &out,
                     const SolverScalars *st, int gate) {
  const MixScan *m = D.scan_of(mix);
  if (!m || in.ls != D.ls) return false;
  const cudaStream_t s = D.lat->stream;
  const int rev = D.lat->turn();
  // up to Ls = 16 and the usual larger ones in registers (FP16 keeps LS / 2
  // outputs too: up to 16 without spills); others read the input twice (FP64,
  // FP32) or take the dense kernels (FP16).  M5^-1 on 16^3x32 in registers /
  // otherwise, Ls = 5, 7, 11, 15: FP64 26 / 31, 33 / 43, 49 / 63, 64 / 87 us,
  // FP32 14 / 14, 18 / 21, 25 / 30, 33 / 39, FP16 12 / 14, 14 / 21, 22 / 39, 33 / 62
  switch (D.ls) {
#define CPSGPU_SCAN_LS(N)                                                                     \
  case N:                                                                                     \
    if (prec == PREC_DOUBLE) launch_full<PREC_DOUBLE, N>(*m, in, out, N, st, gate, s, rev);        \
    else if (prec == PREC_SINGLE) launch_full<PREC_SINGLE, N>(*m, in, out, N, st, gate, s, rev);   \
    else if constexpr (N <= 16) launch_half<N>(*m, in, out, st, gate, s, rev);                     \
    else return false;                                                                        \
    break;
    CPSGPU_SCAN_LS(3)
    CPSGPU_SCAN_LS(4)
    CPSGPU_SCAN_LS(5)
    CPSGPU_SCAN_LS(6)
    CPSGPU_SCAN_LS(7)
    CPSGPU_SCAN_LS(8)
    CPSGPU_SCAN_LS(9)
    CPSGPU_SCAN_LS(10)
    CPSGPU_SCAN_LS(11)
    CPSGPU_SCAN_LS(12)
    CPSGPU_SCAN_LS(13)
    CPSGPU_SCAN_LS(14)
    CPSGPU_SCAN_LS(15)
    CPSGPU_SCAN_LS(16)
    CPSGPU_SCAN_LS(20)
    CPSGPU_SCAN_LS(24)
#undef CPSGPU_SCAN_LS
    default:
      if (prec == PREC_DOUBLE) launch_full<PREC_DOUBLE, 0>(*m, in, out, D.ls, st, gate, s, rev);
      else if (prec == PREC_SINGLE) launch_full<PREC_SINGLE, 0>(*m, in, out, D.ls, st, gate, s, rev);
      else return false;
  }
  CPSGPU_CUDA(cudaGetLastError());
  launch_counter()++;
  return true;
}

}  // namespace cpsgpu
