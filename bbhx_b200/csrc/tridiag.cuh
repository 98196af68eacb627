// Block-cooperative tridiagonal solver shared by the spline build (spline.cu, sparse_build.cu) and
// its adjoint (gradient.cu).
#pragma once

#include "bbhx_common.cuh"

namespace bbhx {

// Cyclic reduction reads rows at strides of powers of two; every array is permuted within its groups
// of 16 doubles (one bank cycle) so that such rows fall into different banks.
__host__ __device__ __forceinline__ int cr_slot(int i) { return i ^ (((i >> 4) ^ (i >> 8)) & 15); }
__host__ __device__ __forceinline__ int cr_pad(int n) { return (n + 15) & ~15; }  // length of an array

// Forward step of cyclic reduction at stride s for row i = 2 s k + 2 s - 1: the matrix, whose two
// multipliers go to w[2 k], w[2 k + 1] for the right-hand sides.
__device__ __forceinline__ void cr_reduce_matrix(double* a, double* b, double* c, double* w, int n,
                                                 int s, int k) {
  const int i = 2 * s * k + 2 * s - 1;
  const int j = cr_slot(i), im = cr_slot(i - s);
  const bool hp = i + s < n;
  const int ip = hp ? cr_slot(i + s) : j;
  const double al = -a[j] / b[im];
  const double ga = hp ? -c[j] / b[ip] : 0.0;
  const double an = al * a[im];
  const double bn = b[j] + al * c[im] + (hp ? ga * a[ip] : 0.0);
  const double cn = hp ? ga * c[ip] : 0.0;
  a[j] = an;
  b[j] = bn;
  c[j] = cn;
  w[2 * k] = al;
  w[2 * k + 1] = ga;
}
__device__ __forceinline__ void cr_reduce_rhs(double* dp, const double* w, int n, int s, int k) {
  const int i = 2 * s * k + 2 * s - 1;
  const int j = cr_slot(i);
  const double al = w[2 * k], ga = w[2 * k + 1];
  const bool hp = i + s < n;
  dp[j] = dp[j] + al * dp[cr_slot(i - s)] + (hp ? ga * dp[cr_slot(i + s)] : 0.0);
}

// In-place cyclic reduction of P right-hand sides d[p * cr_pad(n) + cr_slot(i)] with the matrix
// a, b, c (sub-diagonal, diagonal, super-diagonal, at cr_slot(i)); the solution returns in d, b is
// replaced by its reciprocal.  w: cr_pad(n) doubles of scratch.  All threads of the block
// participate.  The matrix is reduced once per level, by the block while a level has more than 32
// rows, then by one warp; every warp takes right-hand sides of its own, and below the wide levels
// runs them to the end with no barrier.  TEAMS: where the warps are twice the right-hand sides or
// more, a team of W warps shares one: its wide levels take a barrier each, its narrow ones the first warp.
// (One warp for each then left the others idle: 10,000 rows x 1, 300 systems 942 us, 417 with teams,
// 491 with a row's thread walking all quantities.)  Bound by latency: 1024 knots x 9 quantities, six
// systems 40 us, 6144 systems 1.04 ms (two blocks per SM); a row's thread walking all nine through
// conflicting strides, and the levels of 32 rows or fewer left to one warp, took 65 us and 1.40 ms.
template <bool TEAMS>
__device__ inline void cr_solve(double* a, double* b, double* c, double* w, double* d, int P,
                                int n) {
  __shared__ double narrow[2 * 64];  // multipliers of the levels of 32 rows or fewer
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarp = (int)blockDim.x >> 5;
  const int ld = cr_pad(n);
  const int W = TEAMS ? max(1, nwarp / P) : 1;  // warps of a right-hand side's team
  const int nteam = nwarp / W, team = warp / W, sub = warp - team * W;
  int s = 1;
  for (; s < n && n / (2 * s) > 32; s <<= 1) {
    const int cnt = n / (2 * s);
    for (int k = t; k < cnt; k += blockDim.x) cr_reduce_matrix(a, b, c, w, n, s, k);
    __syncthreads();
    for (int p = team; p < P; p += nteam)
      for (int k = sub * 32 + lane; k < cnt; k += 32 * W) cr_reduce_rhs(d + (size_t)p * ld, w, n, s, k);
    __syncthreads();
  }
  const int s0 = s;
  int top = s;
  while (top < n) top <<= 1;
  if (warp == 0) {
    for (int r = s0, o = 0; r < n; r <<= 1) {
      const int cnt = n / (2 * r);
      if (lane < cnt) cr_reduce_matrix(a, b, c, narrow + 2 * o, n, r, lane);
      o += cnt;
      __syncwarp();
    }
  }
  __syncthreads();
  for (int i = t; i < n; i += blockDim.x) b[cr_slot(i)] = 1.0 / b[cr_slot(i)];
  __syncthreads();
  // rows i = r - 1 + 2 r k, k = k0, k0 + step, ..., of a level of the substitution
  auto substitute = [&](double* dp, int r, int cnt, int k0, int step) {
    for (int k = k0; k < cnt; k += step) {
      const int i = r - 1 + 2 * r * k;
      const int j = cr_slot(i);
      const double xm = (i - r >= 0) ? dp[cr_slot(i - r)] : 0.0;
      const double xp = (i + r < n) ? dp[cr_slot(i + r)] : 0.0;
      dp[j] = (dp[j] - a[j] * xm - c[j] * xp) * b[j];
    }
  };
  if (TEAMS && W > 1) {  // one right-hand side per team: the wide levels by all its warps, block by block
    double* dp = d + (size_t)team * ld;
    const bool mine = team < P;
    if (mine && sub == 0)
      for (int r = s0, o = 0; r < n; r <<= 1) {
        const int cnt = n / (2 * r);
        if (lane < cnt) cr_reduce_rhs(dp, narrow + 2 * o, n, r, lane);
        o += cnt;
        __syncwarp();
      }
    for (int r = top; r >= 1; r >>= 1) {
      const int cnt = (n >= r) ? (n - r) / (2 * r) + 1 : 0;
      if (cnt > 32) {
        __syncthreads();
        if (mine) substitute(dp, r, cnt, sub * 32 + lane, 32 * W);
      } else {
        if (mine && sub == 0) substitute(dp, r, cnt, lane, 32);
        __syncwarp();
      }
    }
    __syncthreads();
    return;
  }
  for (int p = warp; p < P; p += nwarp) {
    double* dp = d + (size_t)p * ld;
    for (int r = s0, o = 0; r < n; r <<= 1) {
      const int cnt = n / (2 * r);
      if (lane < cnt) cr_reduce_rhs(dp, narrow + 2 * o, n, r, lane);
      o += cnt;
      __syncwarp();
    }
    for (int r = top; r >= 1; r >>= 1) {
      const int cnt = (n >= r) ? (n - r) / (2 * r) + 1 : 0;
      substitute(dp, r, cnt, lane, 32);
      __syncwarp();
    }
  }
  __syncthreads();
}

}  // namespace bbhx
