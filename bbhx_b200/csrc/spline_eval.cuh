// Shared device helpers for evaluating the nine splined quantities on the data grid.
#pragma once

#include "bbhx_common.cuh"

namespace bbhx {

// The reference's tf gate (WaveformBuild.cu:50): accept when t_start <= tf and
// (tf <= t_end or t_end <= 0).
__device__ __forceinline__ bool tf_gate(double tf, double t_start, double t_end) {
  return (tf >= t_start) && ((tf <= t_end) || (t_end <= 0.0));
}

// t(f) gate over a whole segment from the control points of its cubic (their hull holds it): 1 all
// inside the observation window, 2 all outside, 0 undecided (per-bin gate).
__device__ __forceinline__ int hull_gate(const double* c, double h, double ts, double te) {
  const double a = c[1] * h, q = c[2] * h * h;
  const double p1 = c[0] + a * (1.0 / 3.0);
  const double p2 = c[0] + (2.0 * a + q) * (1.0 / 3.0);
  const double p3 = c[0] + a + q + c[3] * h * h * h;
  const double lo = fmin(fmin(c[0], p1), fmin(p2, p3));
  const double hi = fmax(fmax(c[0], p1), fmax(p2, p3));
  const double eps = 1e-6;  // s: far above the rounding of t(f) (~1e8 s)
  if (!(lo == lo) || !(hi == hi)) return 0;
  if (lo >= ts + eps && (te <= 0.0 || hi <= te - eps)) return 1;
  if (hi < ts - eps || (te > 0.0 && lo > te + eps)) return 2;
  return 0;
}

// conj(T_c * A e^{i phi}) for the three channels (WaveformBuild.cu:48-60)
__device__ __forceinline__ void combine_channels(double amp, double phase, cplx T1, cplx T2,
                                                 cplx T3, cplx& h1, cplx& h2, cplx& h3) {
  double s, c;
  sincos_cw(phase, &s, &c);
  cplx ap = mk(amp * c, amp * s);
  h1 = conj(T1 * ap);
  h2 = conj(T2 * ap);
  h3 = conj(T3 * ap);
}

// Segment of f in the knots xr[0 .. L): searchsorted(right) - 1, guessed for the log-spaced knots
// of the window regrid (per = (L - 1) / log(hi / lo)) and corrected, else by bisection.
__device__ __forceinline__ int segment_guess(const double* __restrict__ xr, int L, double lo,
                                             double hi, float per, double f) {
  if (!(f >= lo)) return -1;
  if (f >= hi) return L - 1;
  int k = (int)(logf((float)(f / lo)) * per);
  k = min(max(k, 0), L - 2);
  for (int it = 0; it < 4; ++it) {
    if (__ldg(xr + k) > f) k = max(k - 1, 0);
    else if (__ldg(xr + k + 1) <= f) k = min(k + 1, L - 2);
    else return k;
  }
  int a = 0, c = L;
  while (a < c) {
    const int mid = (a + c) >> 1;
    if (__ldg(xr + mid) <= f) a = mid + 1; else c = mid;
  }
  return a - 1;
}

// warp-cooperative searchsorted(row, v, side='right') - 1 over a sorted row of length L;
// every lane passes the same v and receives the same result in [-1, L-1].
__device__ __forceinline__ int warp_segment_search(const double* __restrict__ row, int L, double v) {
  int lane = threadIdx.x & 31;
  int lo = 0, hi = L;  // answer count = #{row[j] <= v} lies in [lo, hi]
  while (hi - lo > 32) {
    int step = (hi - lo + 31) / 32;
    int idx = lo + lane * step;
    bool le = (idx < hi) ? (__ldg(row + idx) <= v) : false;
    unsigned m = __ballot_sync(0xffffffffu, le);
    int c = __popc(m);  // lanes 0..c-1 satisfy row[idx] <= v
    if (c == 0) {
      hi = lo;  // v < row[lo] is impossible to refine further: count == lo
      break;
    }
    int nlo = lo + (c - 1) * step + 1;
    int nhi = lo + c * step;
    if (nhi > hi) nhi = hi;
    lo = nlo;
    hi = nhi;
  }
  // final: count = lo + #{j in [lo, hi) : row[j] <= v}
  int idx = lo + lane;
  bool le = (idx < hi) ? (__ldg(row + idx) <= v) : false;
  unsigned m = __ballot_sync(0xffffffffu, le);
  return lo + __popc(m) - 1;
}

}  // namespace bbhx
