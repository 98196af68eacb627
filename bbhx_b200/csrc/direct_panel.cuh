// FP64 direct likelihood on uniform data grids: templates summed panel by panel.
//
// The data bins of a work item are cut into panels: runs of bins that hold no knot of any mode
// and over which the modes' phases stay together.  Over a panel the template of a channel is
//   h_c(i) = conj(Q_c(i) e^{i b (i - ia)}),   Q_c = sum_modes T_c A e^{i (phi - b (i - ia))},
// with one carrier slope b for all modes.  phi' = 2 pi t(f), and at frequencies above a few
// mHz the modes of a massive binary pass a frequency within minutes of each other in an
// observation of months, so the residual phases stay below kPanelDelta over hundreds of bins
// and Q_c is a polynomial of degree 7 to ~5e-14: it is built from the modes' exact values at
// eight nodes (lanes = node x mode), and a bin then costs three polynomials and one carrier
// product for all modes together instead of seven cubics and three rotations per mode (75 FP64
// instructions per bin for six modes, against 306).  Where the modes do not stay together (a
// few 1e-3 of the band) the bins are evaluated one by one.
#pragma once

namespace bbhx {

constexpr int kPanelNodes = 8;
// Residual phase over a panel, linear and quadratic part (rad): the degree-7 interpolation error
// of e^{i (delta s + q s^2)} is ~2e-13 at both limits.  Amplitude and transfer functions add to
// it; panel_smooth checks the coefficients themselves.
constexpr double kPanelDelta = 0.15;
constexpr double kPanelQuad = 1.5e-3;
constexpr float kPanelTail = 1.6e-8f;  // largest |c_6|, |c_7| against the largest coefficient
constexpr int kPanelBins = 1024;       // longest panel
constexpr int kPanelMinBins = 24;      // below this the nodes cost more than the bins
constexpr int kPanelDirect = 128;      // bins evaluated one by one at a time

// Nodes +-t_q on [-1, 1]: Chebyshev points rounded to multiples of 1/128, so that a node's bin
// position is exact.  Row p of kPanelCoef: coefficient of s^p = sum_q row[q] (F(t_q) + F(-t_q))
// for even p, (F(t_q) - F(-t_q)) for odd p.
__device__ const double kPanelTau[4] = {0.984375, 0.828125, 0.5625, 0.1953125};
__device__ const double kPanelCoef[kPanelNodes][4] = {
    {-0.024057555333062423, 0.0863143273345492, -0.188962393279747, 0.6267056212782602},
    {-0.02443942129073008, 0.10422862168700281, -0.3359331436084391, 3.2087327809446924},
    {0.741768143135053, -2.624550413047438, 5.4240838960065085, -3.5413016260941235},
    {0.7535422406451333, -3.169268423302567, 9.642815815122681, -18.13146432560191},
    {-3.0236508244804163, 9.767785072933092, -12.619493021439396, 5.875358772986721},
    {-3.071645282011852, 11.795061220145621, -22.434654260336707, 30.081836917692012},
    {2.906394550207518, -7.380004179614286, 7.454222650728741, -2.980613021321973},
    {2.9525277970362085, -8.91170316028895, 13.251951379073317, -15.260738669168502}};

// Per-warp shared memory of the panel path beside the staged segments.
struct alignas(16) PanelStage {
  double2 C[3][kPanelNodes];   // polynomial coefficients of Q_c in s
  double F[kPanelNodes][6];    // Q_c at the nodes (0..3: +t_q, 4..7: -t_q)
  double lo[FD_MAXM], hi[FD_MAXM];  // first and last knot of each mode
  float per[FD_MAXM];          // (L - 1) / log(hi / lo)
  int kl[FD_MAXM];             // staged segment of each mode in this panel, -1: contributes nothing
};

// First bin i in [0, N] with fl((k0 + i) df) >= x (the grid frequency, see GridInfo).
__device__ __forceinline__ int first_bin_at(double x, double k0, double df, int N) {
  int i = (int)fmin(fmax(ceil(x / df) - k0, 0.0), (double)N);
  while (i > 0 && __dmul_rn(k0 + (double)(i - 1), df) >= x) --i;
  while (i < N && __dmul_rn(k0 + (double)i, df) < x) ++i;
  return i;
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

// Whether the panel's polynomials have converged: the two highest coefficients of every channel
// lie below kPanelTail of its largest one (lanes = channel x power).
__device__ __forceinline__ bool panel_smooth(const PanelStage& PS, int lane) {
  const int ch = min(lane >> 3, 2), p = lane & 7;
  const double2 c = PS.C[ch][p];
  const double v = fabs(c.x) + fabs(c.y);
  double top = v;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  return !__any_sync(0xffffffffu, p >= 6 && v > kPanelTail * top);
}

// Q_c at the panel's nodes, then its polynomial coefficients into PS.C.  Lane = (node, mode
// group): lanes 8 g .. 8 g + 7 take the nodes of modes g and g + 4.  kc = k0 + ia; the node
// sits `off` bins after ia (exact), its phase is evaluated at k df with the error-free product
// and compensated sums of rot_anchor, and the carrier b * off is taken off before the reduction.
__device__ __forceinline__ void panel_nodes(const WarpStage<double>& S, PanelStage& PS, int M,
                                            int lane, double kc, double center, double half,
                                            double df, double b, double tau, const double* row) {
  const int node = lane & 7, grp = lane >> 3;
  const double off = fma(half, tau, center);
  const double kd = kc + off;
  const double p = __dmul_rn(kd, df);
  const double pe = fma(kd, df, -p);
  const double hi = __dmul_rn(b, off);
  const double lo = fma(b, off, -hi);
  double F[6] = {0, 0, 0, 0, 0, 0};
  for (int m = grp; m < M; m += 4) {
    const int k = PS.kl[m];
    if (k < 0) continue;
    const double u = __dsub_rn(p, S.x[m][k]);
    double c[4];
    const SmemCoef src{S, m, k};
    src.get(1, c);
    double t = u * fma(fma(c[3], u, c[2]), u, c[1]);
    t = fma(fma(fma(3.0 * c[3], u, 2.0 * c[2]), u, c[1]), pe, t);
    // c0 + t - hi = sh + se exactly (two TwoSums)
    const double s1 = __dadd_rn(c[0], t);
    const double b1 = __dsub_rn(s1, c[0]);
    const double e1 = __dadd_rn(__dsub_rn(c[0], __dsub_rn(s1, b1)), __dsub_rn(t, b1));
    const double sh = __dsub_rn(s1, hi);
    const double b2 = __dsub_rn(sh, s1);
    const double e2 = __dsub_rn(__dsub_rn(s1, __dsub_rn(sh, b2)), __dadd_rn(hi, b2));
    double sn, cs;
    sincos_cw(sh, &sn, &cs, (e1 + e2) - lo);
    src.get(0, c);
    const double amp = fma(fma(fma(c[3], u, c[2]), u, c[1]), u, c[0]);
    const double apr = amp * cs, api = amp * sn;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      src.get(3 + 2 * ch, c);
      const double tr = fma(fma(fma(c[3], u, c[2]), u, c[1]), u, c[0]);
      src.get(4 + 2 * ch, c);
      const double ti = fma(fma(fma(c[3], u, c[2]), u, c[1]), u, c[0]);
      F[2 * ch] = fma(tr, apr, fma(-ti, api, F[2 * ch]));
      F[2 * ch + 1] = fma(tr, api, fma(ti, apr, F[2 * ch + 1]));
    }
  }
  __syncwarp();
  // sum over the mode groups: the halves exchange three components each, then the quarters
  const bool up = (lane & 16) != 0;
  double v[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const double send = up ? F[q] : F[q + 3];
    const double keep = up ? F[q + 3] : F[q];
    v[q] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], 8);
  if ((lane & 8) == 0) {
    double* dst = &PS.F[node][up ? 3 : 0];
    dst[0] = v[0];
    dst[1] = v[1];
    dst[2] = v[2];
  }
  __syncwarp();
  // coefficient of s^node for components grp and grp + 4
  const double sg = (node & 1) ? -1.0 : 1.0;
  double* C = reinterpret_cast<double*>(PS.C);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int comp = grp + 4 * r;
    if (comp < 6) {
      double a = 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) a = fma(row[q], fma(sg, PS.F[q + 4][comp], PS.F[q][comp]), a);
      C[2 * ((comp >> 1) * kPanelNodes + node) + (comp & 1)] = a;
    }
  }
  __syncwarp();
}

// Sums over the panel's n bins from ia: hh += |w Q|^2, (zr, zi) = sum_i z_i R^(j) of the lane's
// bins i = ia + lane + 32 j, with z = sum_c d~_c w Q_c, taken from the last bin down (Horner in
// R = e^{i 32 b}), so the carrier costs one complex product per bin.
__device__ __forceinline__ void panel_bins(const FusedArgs& A, const PanelStage& PS, int ia, int n,
                                           double center, double inv_half, int lane, double Rr,
                                           double Ri, double& zr, double& zi, double& hh) {
  zr = zi = 0.0;
  const double* wp = A.noise + ia + lane;
  const double2* dp = reinterpret_cast<const double2*>(A.data) + ia + lane;
  for (int j0 = ((n - 1) >> 7) << 2; j0 >= 0; j0 -= FD_K) {
    double s[FD_K], ar[FD_K], ai[FD_K];
    bool ok[FD_K];
#pragma unroll
    for (int j = 0; j < FD_K; ++j) {
      const int i = lane + 32 * (j0 + j);
      ok[j] = i < n;
      s[j] = ok[j] ? ((double)i - center) * inv_half : 0.0;
      ar[j] = 0.0;
      ai[j] = 0.0;
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      double w[FD_K], qr[FD_K], qi[FD_K];
      double2 d[FD_K];
#pragma unroll
      for (int j = 0; j < FD_K; ++j) {
        const long long o = (long long)ch * A.N + 32 * (j0 + j);
        w[j] = ok[j] ? __ldg(wp + o) : 0.0;
        d[j] = ok[j] ? __ldg(dp + o) : make_double2(0.0, 0.0);
      }
      const double2 top = PS.C[ch][kPanelNodes - 1];
#pragma unroll
      for (int j = 0; j < FD_K; ++j) {
        qr[j] = top.x;
        qi[j] = top.y;
      }
#pragma unroll
      for (int p = kPanelNodes - 2; p >= 0; --p) {
        const double2 c = PS.C[ch][p];
#pragma unroll
        for (int j = 0; j < FD_K; ++j) {
          qr[j] = fma(qr[j], s[j], c.x);
          qi[j] = fma(qi[j], s[j], c.y);
        }
      }
#pragma unroll
      for (int j = 0; j < FD_K; ++j) {
        const double hr = qr[j] * w[j], hi = qi[j] * w[j];
        hh = fma(hr, hr, fma(hi, hi, hh));
        ar[j] = fma(d[j].x, hr, fma(-d[j].y, hi, ar[j]));
        ai[j] = fma(d[j].x, hi, fma(d[j].y, hr, ai[j]));
      }
    }
#pragma unroll
    for (int j = FD_K - 1; j >= 0; --j) {
      const double tr = fma(zr, Rr, fma(-zi, Ri, ar[j]));
      zi = fma(zr, Ri, fma(zi, Rr, ai[j]));
      zr = tr;
    }
  }
}

// One bin's template acc (6 reals) times weights and data, into the sums.
__device__ __forceinline__ void bin_products(const FusedArgs& A, int i, const double* acc,
                                             double& dr, double& di, double& hh) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const long long gi = (long long)c * A.N + i;
    const double w = __ldg(A.noise + gi);
    const double2 d = __ldg(reinterpret_cast<const double2*>(A.data) + gi);
    const double hr = acc[2 * c] * w, hi = acc[2 * c + 1] * w;
    dr = fma(d.x, hr, fma(d.y, hi, dr));
    di = fma(d.x, hi, fma(-d.y, hr, di));
    hh = fma(hr, hr, fma(hi, hi, hh));
  }
}

// The n bins from ia one by one (lanes over bins) where the knots lie as close as the bins: every
// bin finds its own segment of each mode and reads the spline arrays.
__device__ __forceinline__ void panel_scatter(const FusedArgs& A, const PanelStage& PS, int b,
                                              int ia, int n, int lane, double k0, double df,
                                              double ts, double te, double& dr, double& di,
                                              double& hh) {
  for (int i = ia + lane; i < ia + n; i += 32) {
    const double f = __dmul_rn(k0 + (double)i, df);
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int m = 0; m < A.M; ++m) {
      const long long o = ((long long)b * A.M + m) * A.L;
      const int k = segment_guess(A.x + o, A.L, PS.lo[m], PS.hi[m], PS.per[m], f);
      if (k >= 0 && k < A.L - 1)
        accumulate_bin_src(GlobalCoef{A, o + k, __ldg(A.x + o + k)}, f, ts, te, acc);
    }
    bin_products(A, i, acc, dr, di, hh);
  }
}

// The n bins from ia one by one (lanes over bins), every mode behind its per-bin t(f) gate: runs
// where a mode crosses the observation window or the modes' phases do not stay together.
__device__ __forceinline__ void panel_direct(const FusedArgs& A, const WarpStage<double>& S,
                                             const PanelStage& PS, int ia, int n, int lane,
                                             double k0, double df, double ts, double te,
                                             double& dr, double& di, double& hh) {
  for (int i = ia + lane; i < ia + n; i += 32) {
    const double f = __dmul_rn(k0 + (double)i, df);
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int m = 0; m < A.M; ++m) {
      const int k = PS.kl[m];
      if (k >= 0) accumulate_bin_src(SmemCoef{S, m, k}, f, ts, te, acc);
    }
    bin_products(A, i, acc, dr, di, hh);
  }
}

// Bins [i0, i1) of binary b (inside its support) by one warp; kk = the segments of bin i0 in
// lanes 0 .. M-1 (-1 before a mode's first knot, L-1 past its last).  Lane m walks mode m: its
// segment, the first bin of the next one, its staged window of segments.  Per-lane partial sums
// into dr, di, hh.
__device__ __forceinline__ void panel_item(const FusedArgs& A, WarpStage<double>& S,
                                           PanelStage& PS, int b, int i0, int i1, int kk,
                                           int lane, double k0, double df, double& dr, double& di,
                                           double& hh) {
  constexpr int NSEG = WarpStage<double>::NSEG;
  const int M = A.M, L = A.L;
  const bool mine = lane < M;
  const double ts = __ldg(A.t_start + b), te = __ldg(A.t_end + b);
  const double tau = (lane & 4) ? -kPanelTau[lane & 3] : kPanelTau[lane & 3];
  double row[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) row[q] = __ldg(&kPanelCoef[lane & 7][q]);
  int k = kk, klo = 0, nst = 0, next = 0;
  int i = i0;
  // runs where the knots of all modes lie closer than kPanelMinBins bins on average
  const double* xr = A.x + ((long long)b * M + (mine ? lane : 0)) * L;
  double lo = 0.0, hi = 0.0;
  float per = 0.0f;
  if (mine) {
    lo = __ldg(xr);
    hi = __ldg(xr + L - 1);
    per = (float)(L - 1) / logf((float)(hi / lo));
    PS.lo[lane] = lo;
    PS.hi[lane] = hi;
    PS.per[lane] = per;
  }
  __syncwarp();
  for (;;) {
    float dens = 0.0f;
    if (mine && k >= 0 && k < L - 1) dens = (float)(df / (__ldg(xr + k + 1) - __ldg(xr + k)));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) dens += __shfl_xor_sync(0xffffffffu, dens, o);
    dens = __shfl_sync(0xffffffffu, dens, 0);
    if (!(dens * (float)kPanelMinBins > 1.0f)) break;
    const int n = min(kPanelDirect, i1 - i);
    panel_scatter(A, PS, b, i, n, lane, k0, df, ts, te, dr, di, hh);
    i += n;
    if (i >= i1) return;
    if (mine) k = segment_guess(xr, L, lo, hi, per, __dmul_rn(k0 + (double)i, df));
  }
  if (mine && k < 0) next = first_bin_at(lo, k0, df, A.N);
  int cap = kPanelBins;  // longest panel that converged of late
  double cb = 0.0, er = 1.0, ei = 0.0, Rr = 1.0, Ri = 0.0;  // carrier slope, e^{i b lane}, e^{32 i b}
  bool fresh = true;  // windows still to be staged
  while (i < i1) {
    // modes whose next knot lies at or before bin i move on; windows they left are staged
    bool move = mine && k < L - 1 && next <= i && !(fresh && k >= 0);
    while (__any_sync(0xffffffffu, move || fresh)) {
      if (move) ++k;
      if (!fresh) cap = min(2 * cap, kPanelBins);
      const bool in = mine && k >= 0 && k < L - 1;
      unsigned need = __ballot_sync(0xffffffffu, in && (k < klo || k >= klo + nst));
      const unsigned staged = need;
      while (need) {
        const int m = __ffs(need) - 1;
        need &= need - 1;
        const int ks = __shfl_sync(0xffffffffu, k, m);
        const int ns = min(NSEG, L - 1 - ks);
        if (lane == m) {
          klo = ks;
          nst = ns;
        }
        stage_segments(A, S, b, m, ks, ns, lane);
      }
      __syncwarp();
      if (staged) {  // whole-segment t(f) gates of the new windows
        const int m = lane >> 2, sg = lane & 3;
        static_assert(NSEG == 4 && FD_MAXM <= 8, "lanes = mode x staged segment");
        const int ns = __shfl_sync(0xffffffffu, nst, m);
        if (((staged >> m) & 1u) && sg < ns)
          S.gate[m][sg] = segment_gate(&S.pc[m][sg][1][0], S.x[m][sg + 1] - S.x[m][sg], ts, te);
        __syncwarp();
      }
      if (in && (move || fresh)) next = first_bin_at(S.x[lane][k + 1 - klo], k0, df, A.N);
      fresh = false;
      move = mine && k < L - 1 && next <= i;
    }
    // bins up to the next knot of any mode; the modes' phase slopes (rad per bin) at both ends
    const bool in = mine && k >= 0 && k < L - 1;
    const int gate = in ? S.gate[lane][k - klo] : 2;
    int e = (mine && k < L - 1) ? next : i1;
    e = __reduce_min_sync(0xffffffffu, e);
    e = min(min(e, i1), i + cap);
    if (mine) PS.kl[lane] = (gate != 2) ? k - klo : -1;
    double mx = -INFINITY, mn = INFINITY, cv = 0.0;
    if (gate != 2) {
      const double* c = &S.pc[lane][k - klo][0][0];
      const double c1 = c[1], c2 = 2.0 * c[2], c3 = 3.0 * c[3], xk = S.x[lane][k - klo];
      const double ua = __dmul_rn(k0 + (double)i, df) - xk;
      const double uz = __dmul_rn(k0 + (double)(e - 1), df) - xk;
      const double sa = fma(fma(c3, ua, c2), ua, c1) * df;
      const double sz = fma(fma(c3, uz, c2), uz, c1) * df;
      mx = fmax(sa, sz);
      mn = fmin(sa, sz);
      cv = mx - mn;
    }
    const unsigned act = __ballot_sync(0xffffffffu, gate != 2);
    const unsigned edge = __ballot_sync(0xffffffffu, gate == 0);
    int n = e - i;
    if (act == 0u) {
      i = e;
      continue;
    }
    __syncwarp();
    if (edge) {
      panel_direct(A, S, PS, i, n, lane, k0, df, ts, te, dr, di, hh);
      __syncwarp();
      i = e;
      continue;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      cv = fmax(cv, __shfl_xor_sync(0xffffffffu, cv, o));
    }
    cv = __shfl_sync(0xffffffffu, cv, 0);
    mx = __shfl_sync(0xffffffffu, mx, 0);
    mn = __shfl_sync(0xffffffffu, mn, 0);
    // residual phase of the panel with a centred carrier: linear 0.25 (mx - mn) n, quadratic
    // cv n / 8 (a slope change of cv over n bins), both shrinking with n
    const double lin = 0.25 * (mx - mn) * n, quad = 0.125 * cv * n;
    if (lin > kPanelDelta || quad > kPanelQuad) {
      const double fit = n * fmin(1.0, fmin(kPanelDelta / lin, sqrt(kPanelQuad / quad)));
      if (fit < kPanelMinBins) {
        n = min(n, kPanelDirect);
        panel_direct(A, S, PS, i, n, lane, k0, df, ts, te, dr, di, hh);
        __syncwarp();
        i += n;
        continue;
      }
      const int pieces = (int)ceil((double)n / fit);
      n = min((n + pieces - 1) / pieces, (int)fit);
    }
    if (!(0.5 * fmax(fabs(mx - cb), fabs(mn - cb)) * n <= kPanelDelta)) {
      cb = 0.5 * (mx + mn);
      sincos_cw(cb * (double)lane, &ei, &er);
      sincos_cw(32.0 * cb, &Ri, &Rr);
    }
    double center, half;
    bool smooth;
    for (;;) {
      center = 0.5 * (double)(n - 1);
      half = fmax(center, 0.5);
      panel_nodes(S, PS, M, lane, k0 + (double)i, center, half, df, cb, tau, row);
      smooth = panel_smooth(PS, lane);
      if (smooth || n <= kPanelMinBins) break;
      n >>= 1;
      cap = n;
    }
    if (!smooth) {
      panel_direct(A, S, PS, i, n, lane, k0, df, ts, te, dr, di, hh);
      __syncwarp();
      i += n;
      continue;
    }
    double zr, zi;
    panel_bins(A, PS, i, n, center, 1.0 / half, lane, Rr, Ri, zr, zi, hh);
    dr = fma(zr, er, fma(-zi, ei, dr));
    di -= fma(zr, ei, zi * er);
    __syncwarp();
    i += n;
  }
}

}  // namespace bbhx
