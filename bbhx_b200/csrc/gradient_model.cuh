// Forward-mode (tangent) parts of the gradient chain: dual-number setup of the per-mode
// PhenomHM and response records, and the contraction of the per-point tangents with the
// adjoint weights produced by the reverse part (heterodyne bin sums or spline adjoint).
//
// Gradient parameters (NGRAD = 11), in this order, with their index in the 12-row
// parameter array of BBHWaveformFD (waveformbuild.py:338-352):
//   0 m1 [Msun] (row 0)   1 m2 [Msun] (1)   2 chi1z (2)   3 chi2z (3)   4 distance [m] (4)
//   5 phi_ref (5)   6 inc (7)   7 lam (8)   8 beta (9)   9 psi (10)   10 t_ref [s] (11)
// f_ref (row 6) does not enter the model (the reference frequency is the amplitude peak).
//
// dL of a point is Re(sum_c u_c dT_c) + phibar dphase + Abar damp with known weights, and the model
// splits: amplitude, phase and t(f) depend on the four intrinsic parameters (and 1 / distance), the
// transfer functions T_c on the angles, through the mode matrix H and the direction k of the
// (binary, mode), and on t = t(f) + t_ref.  So a point takes PhenomHM once with four tangents
// (five where the frequency moves) and the response once forward and once in reverse
// (response_adjoint.cuh), and the angles' tangents meet the summed adjoints of H and k once per
// binary (k_grad_finish).  Bound by FP64 issue and latency at 12 warps per SM.  With all 11 tangents
// carried through the whole model, three at a time in four passes (255 registers, spills, a body
// longer than the instruction cache): 2048 walkers x 6 modes x 128 points 3.3 -> 0.73 ms, 128
// binaries x 6 modes x 512 knots 1.0 -> 0.20 ms.
#pragma once

#include <algorithm>

#include "capi_internal.cuh"
#include "bbhx_common.cuh"
#include "dual.cuh"
#include "phenomhm_model.cuh"
#include "response_adjoint.cuh"
#include "response_model.cuh"
#include "spline_eval.cuh"

namespace bbhx {

constexpr int NGRAD = 11;
constexpr int kIntr = 4;  // m1, m2, chi1z, chi2z
constexpr int kExtr = 5;  // phi_ref, inc, lam, beta, psi
using RD = ad::Dual<kExtr>;

// x with tangent 1 in direction k
template <int N>
__device__ __forceinline__ ad::Dual<N> seed(double v, int k) {
  ad::Dual<N> x(v);
  x.d[k] = 1.0;
  return x;
}

// Records of binaries [b0, b0 + nb) with tangents: blockIdx.y = 0 the PhenomHM record with the
// intrinsic parameters' (ringdown frequencies -> phm_setup_mode; N = 4, or 5 with one direction
// left free for the frequency), 1 the response record with the angles'.  P: the [12, B] parameter
// array; qnm: [8, nq] table y/c1/c2/c3 of the ringdown and damping splines.
template <int N>
static __global__ void k_grad_setup(ModeCoeffsT<ad::Dual<N>>* coeffs, ResponseModeT<RD>* rmodes,
                                    const double* P, int B, int b0, int nb, const int* ells,
                                    const int* mms, int M, const double* qnm, int nq,
                                    double dspin, int run_phenomd) {
  using D = ad::Dual<N>;
  const long long n = (long long)nb * M;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const int bl = (int)(t / M), i = (int)(t % M);
    const int b = b0 + bl;
    auto par = [&](int row) { return P[(size_t)row * B + b]; };
    const int ell = run_phenomd ? 2 : ells[i];
    const int mm = run_phenomd ? 2 : mms[i];
    if (blockIdx.y == 1) {
      response_mode_setup(rmodes[t], ell, mm, seed<kExtr>(par(5), 0), seed<kExtr>(par(7), 1),
                          seed<kExtr>(par(8), 2), seed<kExtr>(par(9), 3), seed<kExtr>(par(10), 4));
      continue;
    }
    const D m1 = seed<N>(par(0), 0), m2 = seed<N>(par(1), 1), chi1 = seed<N>(par(2), 2),
            chi2 = seed<N>(par(3), 3);
    D fm, fs;
    final_mass_spin(m1, m2, chi1, chi2, &fm, &fs);
    // PhenomD 22 ringdown / damping from the tabulated spline (PhenomHMWaveform.cu:1930-1993)
    const int ind = qnm_row(fs.v, dspin, nq - 1);
    const D x = fs - (dspin * ind + (-1.0));
    const D x2 = x * x, x3 = x2 * x;
    const double* y_rd = qnm;
    const double* y_dm = qnm + 4 * (size_t)nq;
    const D rd22 = (y_rd[ind] + y_rd[nq + ind] * x + y_rd[2 * nq + ind] * x2 +
                    y_rd[3 * nq + ind] * x3) / fm;
    const D dm22 = (y_dm[ind] + y_dm[nq + ind] * x + y_dm[2 * nq + ind] * x2 +
                    y_dm[3 * nq + ind] * x3) / fm;
    D rd_lm = rd22, dm_lm = dm22;
    if (!run_phenomd) {
      const cplxT<D> z = qnm_cw(fs, ell, mm);
      rd_lm = (0.5 / PI) * z.re / fm;
      dm_lm = (0.5 / PI) * z.im / fm;
    }
    phm_setup_mode(coeffs[t], m1 * MSUN_SI, m2 * MSUN_SI, chi1, chi2, D(par(4)), ell, mm,
                   rd_lm, dm_lm, rd22, dm22, run_phenomd);
  }
}

// Sums a contraction warp keeps over its points: slots of `part` (one row of 32 per item).
struct PointSums {
  ResponseVec r;                        // 0..14: d L / d (H, k)
  double intr[kIntr];                   // 15..18
  double amp, t;                        // 19: Abar A, 20: d L / d t_ref
  double x_lo, x_hi;                    // 21, 22: d L / d log of the knots' band edges
};
constexpr int kSumIntr = 15, kSumAmp = 19, kSumT = 20, kSumX = 21, kSums = 23;

// m[0..31] of every lane -> lane l returns the warp total of m[l] (recursive halving: at the
// step of width w a lane keeps the half of its w values whose index bit matches its lane bit).
__device__ __forceinline__ double warp_transpose_sum32(double (&m)[32], int lane) {
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    const bool upper = (lane & w) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const double send = upper ? m[i] : m[i + w];
      const double keep = upper ? m[i + w] : m[i];
      m[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return m[0];
}

// A contraction item is a warp's share (part q of Q, every Q-th 32 points) of one (binary, mode):
// all of it where that fills the GPU, else split, to about 16 warps per SM (128 binaries of 6 modes,
// 512 knots: the gradient call takes 8.26 ms split by four, 8.33 unsplit).
inline int contract_split(int nb, int M, int L) {
  const long long rows = (long long)nb * M, want = 16ll * sm_count();
  return (int)std::max(1ll, std::min((want + rows - 1) / rows, (long long)(L + 31) / 32));
}
constexpr int kContractWarps = 4;
inline unsigned contract_blocks(int nb, int M, int Q) {
  const long long blocks = ((long long)nb * M * Q + kContractWarps - 1) / kContractWarps;
  return (unsigned)std::min(blocks, (long long)sm_count() * 32);
}

// Contraction of the model's tangents with the adjoint weights, summed over the points of an item
// into part[item][32] (k_grad_finish).
//   DIRECT = false, heterodyned: weights gh[c, j] of the sparse grid `freqs`, dL = Re(gh dW) with
//     W_c = T_c A e^{i phase} (lnL depends on h = sum_modes conj(W)).
//   DIRECT = true: weights ybar of the [9, B, M, L] spline buffer (amplitude, phase with t_ref
//     shift and Roemer delay, the six transfer components; t(f) only gates) and xbar of the knots
//     x = flo^(1 - r) fhi^r, r = i / (L - 1), which move with the observation-window regrid: the
//     quantities are differentiated along the moving knot, the frequency being the fifth tangent.
template <bool DIRECT>
struct ContractArgs {
  double* part;
  const ModeCoeffsT<ad::Dual<DIRECT ? kIntr + 1 : kIntr>>* coeffs;
  const ResponseModeT<RD>* rmodes;
  OrbitTables orb;
  const double* P;
  int B, b0, nb;
  double t_init;
  const double *t_start, *t_end, *freqs;  // heterodyned
  const cplx* gh;
  const double *x, *ybar, *xbar;          // direct
  int TDItag, rescaled, tdi2, M, L, Q;
};

// Heterodyned, three CTAs per SM at 168 registers: 2048 walkers' call takes 1.14 ms, 1.19 with two
// (255), 1.17 with four (128); the direct form, longer by the frequency's tangent, takes two.
template <bool DIRECT>
static __global__ void __launch_bounds__(kContractWarps * 32, DIRECT ? 2 : 3)
k_contract(ContractArgs<DIRECT> A) {
  using D = ad::Dual<DIRECT ? kIntr + 1 : kIntr>;
  __shared__ ResponseVec rv[kContractWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int L = A.L, M = A.M;
  const long long total = (long long)A.nb * M * A.Q;
  const size_t n = (size_t)A.B * M * L;
  for (long long it = blockIdx.x * (long long)kContractWarps + wid; it < total;
       it += (long long)gridDim.x * kContractWarps) {
    const int rec = (int)(it / A.Q), q0 = (int)(it - (long long)rec * A.Q);
    const int b = A.b0 + rec / M, m = rec % M;
    const ModeCoeffsT<D>& c = A.coeffs[rec];
    ResponseVec& r = rv[wid];
    __syncwarp();
    {
      const ResponseModeT<RD>& g = A.rmodes[rec];
      if (lane < 6) {
        r.re[lane] = g.H[sym_index(lane)].re.v;
        r.im[lane] = g.H[sym_index(lane)].im.v;
      }
      if (lane < 3) r.k[lane] = g.k[lane].v;
    }
    __syncwarp();
    const double t_ref = A.P[11 * (size_t)A.B + b];
    PointSums s = {};
    for (int j = q0 * 32 + lane; j < L; j += 32 * A.Q) {
      if constexpr (!DIRECT) {
        const double f = A.freqs[j];
        const PointOutT<D> w = phm_eval_point(c, D(f));
        const double t = w.tf.v + t_ref;
        if (!tf_gate(t, A.t_start[b], A.t_end[b])) continue;
        RoemerPoint rp;
        const double R = roemer(r, f, t, &rp);
        const cplx e = expi(w.phase.v + (2 * PI * f) * (t_ref - A.t_init) + R);
        cplx u[3];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch)
          u[ch] = w.amp.v * (A.gh[((size_t)b * 3 + ch) * L + j] * e);
        double tbar = 0.0, fbar = 0.0;
        const cplx ut = links_adjoint<false>(r, A.orb, f, t, u, A.TDItag, A.rescaled, A.tdi2, s.r,
                                             &tbar, &fbar);
        const double abar = w.amp.v != 0.0 ? ut.re / w.amp.v : 0.0, phibar = -ut.im;
        roemer_adjoint(r, rp, phibar, s.r, &tbar);
#pragma unroll
        for (int k = 0; k < kIntr; ++k)
          s.intr[k] += abar * w.amp.d[k] + phibar * w.phase.d[k] + tbar * w.tf.d[k];
        s.amp += ut.re;
        s.t += tbar + phibar * (2 * PI * f);
      } else {
        const size_t o = ((size_t)b * M + m) * L + j;
        const double abar = A.ybar[o], phibar = A.ybar[n + o], xb = A.xbar[o];
        cplx u[3];  // Re(u dT) = wr d Re T + wi d Im T
        bool any = abar != 0.0 || phibar != 0.0 || xb != 0.0;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
          u[ch] = cmk(A.ybar[(size_t)(3 + 2 * ch) * n + o], -A.ybar[(size_t)(4 + 2 * ch) * n + o]);
          any = any || u[ch].re != 0.0 || u[ch].im != 0.0;
        }
        if (!any) continue;
        const double f = A.x[o];
        const PointOutT<D> w = phm_eval_point(c, seed<kIntr + 1>(f, kIntr));
        const double t = w.tf.v + t_ref;
        RoemerPoint rp;
        const double R = roemer(r, f, t, &rp);
        double tbar = 0.0, fbar = xb + phibar * (2 * PI * (t_ref - A.t_init) + R / f);
        links_adjoint<true>(r, A.orb, f, t, u, A.TDItag, A.rescaled, A.tdi2, s.r, &tbar, &fbar);
        roemer_adjoint(r, rp, phibar, s.r, &tbar);
#pragma unroll
        for (int k = 0; k < kIntr; ++k)
          s.intr[k] += abar * w.amp.d[k] + phibar * w.phase.d[k] + tbar * w.tf.d[k];
        fbar += abar * w.amp.d[kIntr] + phibar * w.phase.d[kIntr] + tbar * w.tf.d[kIntr];
        s.amp += abar * w.amp.v;
        s.t += tbar + phibar * (2 * PI * f);
        const double xr = j / (double)(L - 1);
        s.x_lo += fbar * f * (1.0 - xr);
        s.x_hi += fbar * f * xr;
      }
    }
    double v[32];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      v[i] = s.r.re[i];
      v[6 + i] = s.r.im[i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) v[12 + i] = s.r.k[i];
#pragma unroll
    for (int i = 0; i < kIntr; ++i) v[kSumIntr + i] = s.intr[i];
    v[kSumAmp] = s.amp;
    v[kSumT] = s.t;
    v[kSumX] = s.x_lo;
    v[kSumX + 1] = s.x_hi;
#pragma unroll
    for (int i = kSums; i < 32; ++i) v[i] = 0.0;
    A.part[it * 32 + lane] = warp_transpose_sum32(v, lane);
  }
}

// Rows of wreg: d log flo, d log fhi of a (binary, mode) for m1, m2, chi1z, chi2z, lam, beta, t_ref
constexpr int kReg = 7;

// grad [B, 11] of binaries [b0, b0 + nb) from the items' sums: those of H and k meet the angles'
// tangents of the records, those of the band edges the regrid's (wreg, null: knots held fixed).
// One warp per binary, a lane per slot (a thread per parameter walked 24 dependent rows).
static __global__ void k_grad_finish(double* grad, const double* part,
                                     const ResponseModeT<RD>* rmodes, const double* wreg,
                                     const double* P, int B, int b0, int nb, int M, int Q) {
  const int lane = threadIdx.x & 31;
  const int nw = (int)(gridDim.x * blockDim.x) >> 5;
  for (int bl = (int)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; bl < nb; bl += nw) {
    double sum = 0.0, ext[kExtr] = {}, reg[kReg] = {};
    for (int m = 0; m < M; ++m) {
      const size_t rec = (size_t)bl * M + m;
      double v = 0.0;
      for (int q = 0; q < Q; ++q) v += part[(rec * Q + q) * 32 + lane];
      sum += v;
      if (lane < kSumIntr) {
        const ResponseModeT<RD>& r = rmodes[rec];
        const RD& g = lane < 6 ? r.H[sym_index(lane)].re
                               : (lane < 12 ? r.H[sym_index(lane - 6)].im : r.k[lane - 12]);
#pragma unroll
        for (int k = 0; k < kExtr; ++k) ext[k] += v * g.d[k];
      }
      if (wreg != nullptr && (lane == kSumX || lane == kSumX + 1)) {
        const double* w = wreg + (rec * 2 + (lane - kSumX)) * kReg;
#pragma unroll
        for (int k = 0; k < kReg; ++k) reg[k] += v * w[k];
      }
    }
#pragma unroll
    for (int k = 0; k < kExtr; ++k)
      for (int o = 16; o > 0; o >>= 1) ext[k] += __shfl_xor_sync(0xffffffffu, ext[k], o);
#pragma unroll
    for (int k = 0; k < kReg; ++k)
      reg[k] = __shfl_sync(0xffffffffu, reg[k], kSumX) + __shfl_sync(0xffffffffu, reg[k], kSumX + 1);
    double* g = grad + (size_t)(b0 + bl) * NGRAD;
    const int ki = lane - kSumIntr;
#pragma unroll
    for (int k = 0; k < kIntr; ++k)
      if (ki == k) g[k] = sum + reg[k];
    if (lane == kSumAmp) g[4] = -sum / P[4 * (size_t)B + b0 + bl];
    if (lane == kSumT) g[10] = sum + reg[6];
    if (lane == 0) {
      g[5] = ext[0];
      g[6] = ext[1];
      g[7] = ext[2] + reg[4];
      g[8] = ext[3] + reg[5];
      g[9] = ext[4];
    }
  }
}

}  // namespace bbhx
