// FP64 direct likelihood on uniform data grids: templates summed panel by panel.
//
// The data bins of a work item are cut into panels: runs of bins that hold no knot of any mode
// and over which the modes' phases stay together.  Over a panel the template of a channel is
//   h_c(i) = conj(Q_c(i) e^{i b (i - ia)}),   Q_c = sum_modes T_c A e^{i (phi - b (i - ia))},
// with one carrier slope b for all modes.  phi' = 2 pi t(f), and at frequencies above a few
// mHz the modes of a massive binary pass a frequency within minutes of each other in an
// observation of months, so the residual phases stay below kPanelDelta over hundreds of bins
// and Q_c is a polynomial of degree 7 to 2.3e-12 of its largest value at worst (kPanelTail): it is
// built from the modes' exact values at eight nodes (lanes = node x mode), and a bin then costs three polynomials and one carrier
// product for all modes together instead of seven cubics and three rotations per mode: 101 FP64
// instructions per bin for six modes with everything included, against 306.  Where the modes do
// not stay together (1-4 % of the band of a 1-yr stream) the bins are evaluated one by one.
//
// What bounds it (B = 1024, 1 yr, six modes, L = 1024; 86.4 ms before the panels, 27 ms now): the
// FP64 pipe is 50 % busy counted at 2 cycles an instruction, but a DFMA that reads three
// registers anew takes 3 (40.7 of 64 lanes per clock measured, 53 in the order of panel_bins), so
// the pipe is two thirds busy, the shared-memory and load path 60 %, issue 50 %.  Data in L1
// instead of L2: no change.  A second resident CTA's worth of warps (16 per SM at 128 registers)
// gains 3 % on large batches and loses 5 % on small ones; dropping negligible powers at run time,
// unrolled per degree or in a short loop over channels: 3-5 % slower.
#pragma once

namespace bbhx {

constexpr int kPanelNodes = 8;
// Residual phase over a panel, linear and quadratic part (rad): the degree-7 interpolation error
// of e^{i (delta s + q s^2)} alone is ~2e-13 at both limits.  Amplitude and transfer functions add
// to it; panel_smooth checks the coefficients themselves: with c_6 and c_7 below kPanelTail of the
// largest, the next is below kPanelDelta / 8 of that, 3e-10, and its remainder 2^-7 of it, 2.3e-12.
// Measured against 80-bit sums: <h|h> of spline sets of 256 to 1000 knots over 0.2 to 1 year to 2e-13
// and better.
constexpr float kPanelDelta = 0.15f;
constexpr float kPanelQuad = 1.5e-3f;
constexpr float kPanelTail = 1.6e-8f;  // largest |c_6|, |c_7| against the largest coefficient
constexpr int kPanelBins = 1024;       // longest panel
constexpr int kPanelMinBins = 24;      // below this the nodes cost more than the bins
constexpr int kPanelDirect = 128;      // bins evaluated one by one at a time
constexpr int kPanelRing = 4;          // segments of a mode in shared memory (power of two)

// Nodes +-t_q on [-1, 1]: Chebyshev points rounded to multiples of 1/128, so that a node's bin
// position is exact.  Row p of kPanelCoef: coefficient of s^p = sum_q row[q] (F(t_q) + F(-t_q))
// for even p, (F(t_q) - F(-t_q)) for odd p.
__device__ const double kPanelTau[4] = {0.984375, 0.828125, 0.5625, 0.1953125};
__device__ const __align__(16) double kPanelCoef[kPanelNodes][4] = {
    {-0.024057555333062423, 0.0863143273345492, -0.188962393279747, 0.6267056212782602},
    {-0.02443942129073008, 0.10422862168700281, -0.3359331436084391, 3.2087327809446924},
    {0.741768143135053, -2.624550413047438, 5.4240838960065085, -3.5413016260941235},
    {0.7535422406451333, -3.169268423302567, 9.642815815122681, -18.13146432560191},
    {-3.0236508244804163, 9.767785072933092, -12.619493021439396, 5.875358772986721},
    {-3.071645282011852, 11.795061220145621, -22.434654260336707, 30.081836917692012},
    {2.906394550207518, -7.380004179614286, 7.454222650728741, -2.980613021321973},
    {2.9525277970362085, -8.91170316028895, 13.251951379073317, -15.260738669168502}};

// Per-warp shared memory of the panel path.  Segment k of mode m (9 quantities x (y, c1, c2, c3))
// sits in ring slot k mod 4, knot j in slot j mod 8.
struct alignas(16) PanelStage {
  double co[FD_MAXM][kPanelRing][FD_NC];
  double x[FD_MAXM][8];
  double2 C[3][kPanelNodes];   // polynomial coefficients of Q_c in s
  double F[kPanelNodes][6];    // Q_c at the nodes (0..3: +t_q, 4..7: -t_q)
  double2 E[32];               // e^{i b lane}
  double xk[FD_MAXM];          // knot of each mode's segment in this panel
  double kb[FD_MAXM];          // its position in bins
  float4 sl[FD_MAXM];          // phase slope in rad per bin, x + y t + z t^2 at t bins after it
  double lo[FD_MAXM], hi[FD_MAXM];  // first and last knot of each mode
  float per[FD_MAXM];          // (L - 1) / log(hi / lo)
  int slot[FD_MAXM];           // ring slot of each mode's segment, -1: contributes nothing
};

// Quantity p (0 amplitude, 1 phase, 2 t(f), 3..8 transfer) of a staged segment.
struct PanelCoef {
  const double* seg;
  double x;
  __device__ __forceinline__ double xk() const { return x; }
  __device__ __forceinline__ void get(int p, double* c) const {
    const double2 lo = *reinterpret_cast<const double2*>(seg + 4 * p);
    const double2 hi = *reinterpret_cast<const double2*>(seg + 4 * p + 2);
    c[0] = lo.x; c[1] = lo.y; c[2] = hi.x; c[3] = hi.y;
  }
};

// 8 bytes from global to shared memory without a register in between.
__device__ __forceinline__ void copy8_async(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// First bin i in [0, N] with fl((k0 + i) df) >= x (the grid frequency, see GridInfo), from the
// knot's position xb = x / df - k0 in bins (good to ~1e-9: only near an integer the frequencies
// themselves are compared).
__device__ __forceinline__ int first_bin_at(double x, double xb, double k0, double df, int N) {
  const double c = ceil(xb);
  int i = (int)fmin(fmax(c, 0.0), (double)N);
  if (!(fabs(xb - rint(xb)) > 1e-6)) {
    while (i > 0 && __dmul_rn(k0 + (double)(i - 1), df) >= x) --i;
    while (i < N && __dmul_rn(k0 + (double)i, df) < x) ++i;
  }
  return i;
}

// Order-preserving integer of a float and back (warp max / min by integer reductions).
__device__ __forceinline__ int order_key(float v) {
  const int b = __float_as_int(v);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float order_value(int k) {
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}

// Whether the panel's polynomials have converged: the two highest coefficients of every channel
// lie below kPanelTail of its largest one (lanes = channel x power).
__device__ __forceinline__ bool panel_smooth(const PanelStage& PS, int lane) {
  const double2 c = PS.C[min(lane >> 3, 2)][lane & 7];
  const float v = (float)(fabs(c.x) + fabs(c.y));
  float top = v;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  return !__any_sync(0xffffffffu, (lane & 7) >= 6 && v > kPanelTail * top);
}

// Q_c at the panel's nodes, then its polynomial coefficients into PS.C.  Lane = (node, mode
// group): lanes 8 g .. 8 g + 7 take the nodes of modes g and g + 4.  kc = k0 + ia; the node
// sits `off` bins after ia (exact), its phase is evaluated at k df with the error-free product
// and compensated sums of rot_anchor, and the carrier b * off is taken off before the reduction.
__device__ __forceinline__ void panel_nodes(PanelStage& PS, int M, int lane, double kc,
                                            double center, double half, double df, double b) {
  const int node = lane & 7, grp = lane >> 3;
  const double tau = (lane & 4) ? -kPanelTau[lane & 3] : kPanelTau[lane & 3];
  const double off = fma(half, tau, center);
  const double kd = kc + off;
  const double p = __dmul_rn(kd, df);
  const double pe = fma(kd, df, -p);
  const double hi = __dmul_rn(b, off);
  const double lo = fma(b, off, -hi);
  double F[6] = {0, 0, 0, 0, 0, 0};
  for (int m = grp; m < M; m += 4) {
    const int sl = PS.slot[m];
    if (sl < 0) continue;
    const PanelCoef src{PS.co[m][sl], PS.xk[m]};
    const double u = __dsub_rn(p, src.x);
    const double ue = __dadd_rn(__dsub_rn(__dsub_rn(p, u), src.x), pe);  // u + ue = k df - x_k
    double c[4];
    src.get(1, c);
    // t + te = u (c1 + c2 u + c3 u^2) + phi'(u) ue: t reaches 4e5 rad in the widest segments, where
    // its rounding alone would be 3e-11 rad at every node, of its own at each
    const double a = __dmul_rn(c[2], u);
    const double ae = fma(__dmul_rn(c[3], u), u, fma(c[2], u, -a));
    const double v = __dadd_rn(c[1], a);
    const double bv = __dsub_rn(v, c[1]);
    const double ve = __dadd_rn(__dsub_rn(c[1], __dsub_rn(v, bv)), __dsub_rn(a, bv)) + ae;
    const double t = __dmul_rn(u, v);
    const double te = fma(u, ve, fma(fma(fma(3.0 * c[3], u, 2.0 * c[2]), u, c[1]), ue,
                                     fma(u, v, -t)));
    // c0 + t - hi = sh + se exactly (two TwoSums)
    const double s1 = __dadd_rn(c[0], t);
    const double b1 = __dsub_rn(s1, c[0]);
    const double e1 = __dadd_rn(__dsub_rn(c[0], __dsub_rn(s1, b1)), __dsub_rn(t, b1));
    const double sh = __dsub_rn(s1, hi);
    const double b2 = __dsub_rn(sh, s1);
    const double e2 = __dsub_rn(__dsub_rn(s1, __dsub_rn(sh, b2)), __dadd_rn(hi, b2));
    double sn, cs;
    sincos_cw(sh, &sn, &cs, ((e1 + e2) - lo) + te);
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
  const double2 r01 = __ldg(reinterpret_cast<const double2*>(kPanelCoef[node]));
  const double2 r23 = __ldg(reinterpret_cast<const double2*>(kPanelCoef[node]) + 1);
  const double row[4] = {r01.x, r01.y, r23.x, r23.y};
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

// Sums over the panel's n bins from ia: hh += |w Q|^2, (zr, zi) = sum_j a_j R^j over the lane's
// bins i = ia + lane + 32 j, a = sum_c d~_c w Q_c, taken from the last bin down (Horner in
// R = e^{i 32 b}), so the carrier costs one complex product per bin.
__device__ __forceinline__ void panel_bins(const FusedArgs& A, const PanelStage& PS, int ia, int n,
                                           double center, double inv_half, int lane, double Rr,
                                           double Ri, double& zr, double& zi, double& hh) {
  zr = zi = 0.0;
  const double* wp = A.noise + ia + lane;
  const double2* dp = reinterpret_cast<const double2*>(A.data) + ia + lane;
  const double s0 = ((double)lane - center) * inv_half, ds = 32.0 * inv_half;
  for (int j0 = ((n - 1) >> 7) << 2; j0 >= 0; j0 -= FD_K) {
    const bool full = n - 32 * j0 >= 32 * FD_K;  // every lane has all its bins
    double s[FD_K], ar[FD_K], ai[FD_K];
#pragma unroll
    for (int j = 0; j < FD_K; ++j) {
      s[j] = fma((double)(j0 + j), ds, s0);
      ar[j] = 0.0;
      ai[j] = 0.0;
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      double w[FD_K], qr[FD_K], qi[FD_K];
      double2 d[FD_K];
      const double* wc = wp + (long long)ch * A.N + 32 * j0;
      const double2* dc = dp + (long long)ch * A.N + 32 * j0;
      if (full) {
#pragma unroll
        for (int j = 0; j < FD_K; ++j) {
          w[j] = __ldg(wc + 32 * j);
          d[j] = __ldg(dc + 32 * j);
        }
      } else {
#pragma unroll
        for (int j = 0; j < FD_K; ++j) {
          const bool ok = lane + 32 * (j0 + j) < n;
          w[j] = ok ? __ldg(wc + 32 * j) : 0.0;
          d[j] = ok ? __ldg(dc + 32 * j) : make_double2(0.0, 0.0);
        }
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
        for (int j = 0; j < FD_K; ++j) qr[j] = fma(qr[j], s[j], c.x);
#pragma unroll
        for (int j = 0; j < FD_K; ++j) qi[j] = fma(qi[j], s[j], c.y);
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

template <bool GH>
__device__ __forceinline__ void bin_products(const FusedArgs& A, cplx* gh, int i, const double* acc,
                                             double& dr, double& di, double& hh);

// panel_bins for the gradient: the same sums and d lnL / d h = 4 w (d~ - w h) of every bin, which
// needs the carrier e^{i b (i - ia)} bin by bin (rotated along the lane's bins).
__device__ __forceinline__ void panel_bins_gh(const FusedArgs& A, cplx* gh, const PanelStage& PS,
                                              int ia, int n, double center, double inv_half,
                                              int lane, double Rr, double Ri, double& dr,
                                              double& di, double& hh) {
  const double s0 = ((double)lane - center) * inv_half, ds = 32.0 * inv_half;
  const double2 E = PS.E[lane];
  double er = E.x, ei = E.y;
  for (int i = lane, j = 0; i < n; i += 64, j += 2) {
    double f[2][6], s[2], cr[2], ci[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      s[t] = fma((double)(j + t), ds, s0);
      cr[t] = er;
      ci[t] = ei;
      cmul_inplace(er, ei, Rr, Ri);
    }
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      double qr[2], qi[2];
      const double2 top = PS.C[ch][kPanelNodes - 1];
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        qr[t] = top.x;
        qi[t] = top.y;
      }
#pragma unroll
      for (int p = kPanelNodes - 2; p >= 0; --p) {
        const double2 c = PS.C[ch][p];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          qr[t] = fma(qr[t], s[t], c.x);
          qi[t] = fma(qi[t], s[t], c.y);
        }
      }
#pragma unroll
      for (int t = 0; t < 2; ++t) {  // h = conj(Q e^{i c})
        f[t][2 * ch] = fma(qr[t], cr[t], -qi[t] * ci[t]);
        f[t][2 * ch + 1] = -fma(qr[t], ci[t], qi[t] * cr[t]);
      }
    }
    bin_products<true>(A, gh, ia + i, f[0], dr, di, hh);
    if (i + 32 < n) bin_products<true>(A, gh, ia + i + 32, f[1], dr, di, hh);
  }
}

// One bin's template acc (6 reals) times weights and data, into the sums; GH: and its d lnL / d h =
// 4 w (d~ - w h) to gh[3 i + channel] (gh addressed by data bin).
template <bool GH>
__device__ __forceinline__ void bin_products(const FusedArgs& A, cplx* gh, int i, const double* acc,
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
    if (GH) gh[3LL * i + c] = mk(4.0 * w * (d.x - hr), 4.0 * w * (d.y - hi));
  }
}

// The n bins from ia one by one (lanes over bins) where the knots lie as close as the bins: every
// bin finds its own segment of each mode and reads the spline arrays.
template <bool GH>
__device__ __forceinline__ void panel_scatter(const FusedArgs& A, cplx* gh, const PanelStage& PS,
                                              int b, int ia, int n, int lane, double k0, double df,
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
    bin_products<GH>(A, gh, i, acc, dr, di, hh);
  }
}

// The n bins from ia one by one, G bins per lane at a time: runs where a mode crosses the
// observation window (GATE: its t(f) decides bin by bin) or the modes' phases do not stay
// together.
template <int G, bool GATE, bool GH>
__device__ __forceinline__ void panel_direct(const FusedArgs& A, cplx* gh, const PanelStage& PS, int b,
                                             int ia, int n, int lane, double k0, double df,
                                             double& dr, double& di, double& hh) {
  double ts = 0.0, te = 0.0;
  if (GATE) {
    ts = __ldg(A.t_start + b);
    te = __ldg(A.t_end + b);
  }
#pragma unroll 1
  for (int i = lane; i < n; i += 32 * G) {
    double f[G], acc[G][6];
#pragma unroll
    for (int j = 0; j < G; ++j) {
      f[j] = __dmul_rn(k0 + (double)(ia + min(i + 32 * j, n - 1)), df);
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[j][c] = 0.0;
    }
#pragma unroll 1
    for (int m = 0; m < A.M; ++m) {
      const int sl = PS.slot[m];
      if (sl < 0) continue;
      const PanelCoef src{PS.co[m][sl], PS.xk[m]};
      double c[4], u[G], apr[G], api[G];
      bool in[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        u[j] = f[j] - src.x;
        in[j] = true;
      }
      if (GATE) {
        src.get(2, c);
#pragma unroll
        for (int j = 0; j < G; ++j)
          in[j] = tf_gate(fma(fma(fma(c[3], u[j], c[2]), u[j], c[1]), u[j], c[0]), ts, te);
      }
      src.get(1, c);
#pragma unroll
      for (int j = 0; j < G; ++j)
        sincos_cw(fma(fma(fma(c[3], u[j], c[2]), u[j], c[1]), u[j], c[0]), &api[j], &apr[j]);
      src.get(0, c);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const double a = in[j] ? fma(fma(fma(c[3], u[j], c[2]), u[j], c[1]), u[j], c[0]) : 0.0;
        apr[j] *= a;
        api[j] *= a;
      }
#pragma unroll
      for (int ch = 0; ch < 3; ++ch) {
        src.get(3 + 2 * ch, c);
        double e[4];
        src.get(4 + 2 * ch, e);
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const double tr = fma(fma(fma(c[3], u[j], c[2]), u[j], c[1]), u[j], c[0]);
          const double ti = fma(fma(fma(e[3], u[j], e[2]), u[j], e[1]), u[j], e[0]);
          acc[j][2 * ch] += tr * apr[j] - ti * api[j];
          acc[j][2 * ch + 1] -= tr * api[j] + ti * apr[j];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < G; ++j)
      if (i + 32 * j < n) bin_products<GH>(A, gh, ia + i + 32 * j, acc[j], dr, di, hh);
  }
  __syncwarp();
}

// Bins [i0, i1) of binary b (inside its support, i0 < i1) by one warp; kk = the segments of bins i0 and
// i1 - 1 in lanes 0 .. M-1 (-1 before a mode's first knot, L-1 past its last).  Lane m walks mode
// m.  When a mode enters segment k its freed ring slot is refilled with segment k + 3 by
// asynchronous copies, three entries ahead of their use.  Per-lane partial sums into dr, di, hh;
// GH: also d lnL / d h of every bin to A.gh (gradient chain).
template <bool GH>
__device__ __forceinline__ void panel_item(const FusedArgs& A, PanelStage& PS, int b, int i0,
                                           int i1, int2 kk, int lane, double k0, double df,
                                           double& dr, double& di, double& hh) {
  const int M = A.M, L = A.L;
  cplx* gh = nullptr;
  if (GH) gh = A.gh + 3 * (__ldg(A.gh_off + b) - (long long)__ldg(A.sup_start + b));
  const bool mine = lane < M;
  int k = mine ? kk.x : L - 1;
  const int klast = mine ? min(kk.y, L - 2) : -1;  // last segment of the item
  int i = i0;
  // runs where the knots of all modes lie closer than kPanelMinBins bins on average
  if (__reduce_add_sync(0xffffffffu, mine ? kk.y - kk.x : 0) * kPanelMinBins > i1 - i0) {
    const double ts = __ldg(A.t_start + b), te = __ldg(A.t_end + b);
    const double* xr = A.x + ((long long)b * M + (mine ? lane : 0)) * L;
    const double lo = __ldg(xr), hi = __ldg(xr + L - 1);
    const float per = (float)(L - 1) / logf((float)(hi / lo));
    if (mine) {
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
      panel_scatter<GH>(A, gh, PS, b, i, n, lane, k0, df, ts, te, dr, di, hh);
      i += n;
      if (i >= i1) return;
      if (mine) k = segment_guess(xr, L, lo, hi, per, __dmul_rn(k0 + (double)i, df));
    }
  }
  // segment seg of mode m and the knot after it: this lane's element (quantity lane / 4,
  // coefficient lane mod 4), lanes 0..3 also element 32 + lane of the ninth quantity
  auto fetch = [&](int m, int seg) {
    double* dst = PS.co[m][seg & (kPanelRing - 1)];
    const long long o = ((long long)b * M + m) * L + seg;
    const int cc = lane & 3;
    const double* src = ((cc == 0) ? A.y : (cc == 1) ? A.c1 : (cc == 2) ? A.c2 : A.c3) + o;
    copy8_async(dst + lane, src + (lane >> 2) * A.qstride);
    if (lane < 4) copy8_async(dst + 32 + lane, src + 8 * A.qstride);
    if (lane == 4) copy8_async(&PS.x[m][(seg + 1) & 7], A.x + o + 1);
  };
  for (int m = 0; m < M; ++m) {
    const int ks = max(__shfl_sync(0xffffffffu, k, m), 0);
    const int kz = min(__shfl_sync(0xffffffffu, klast, m), ks + kPanelRing - 1);
    if (lane == 5 && ks <= kz) copy8_async(&PS.x[m][ks & 7], A.x + ((long long)b * M + m) * L + ks);
    for (int s = ks; s <= kz; ++s) fetch(m, s);
  }
  copy_commit();
  copy_wait<0>();
  __syncwarp();
  // per-lane state of mode `lane`: segment k, first bin of the next one, gate (2: nothing to add)
  int next = 0, gate = 2;
  auto enter = [&]() {  // lane's mode has arrived in segment k
    gate = 2;
    if (k < L - 1) {
      const double x1 = PS.x[lane][(k + 1) & 7];
      const double inv_df = 1.0 / df;
      const double xb1 = fma(x1, inv_df, -k0);
      next = first_bin_at(x1, xb1, k0, df, A.N);
      if (k >= 0) {
        const double* c = PS.co[lane][k & (kPanelRing - 1)];
        const double x0 = PS.x[lane][k & 7];
        gate = hull_gate(c + 8, x1 - x0, __ldg(A.t_start + b), __ldg(A.t_end + b));
        PS.kb[lane] = fma(x0, inv_df, -k0);
        PS.sl[lane] = make_float4((float)(c[5] * df), (float)(2.0 * c[6] * df * df),
                                  (float)(3.0 * c[7] * df * df * df), 0.0f);
        PS.xk[lane] = x0;
      }
    }
    PS.slot[lane] = (gate != 2) ? (k & (kPanelRing - 1)) : -1;
  };
  if (mine) {
    if (k < 0) {  // before the mode's first knot: wait for it
      next = i1;
      if (klast >= 0) {
        const double x0 = PS.x[lane][0];
        next = first_bin_at(x0, x0 / df - k0, k0, df, A.N);
      }
      PS.slot[lane] = -1;
    } else {
      enter();
    }
  }
  int cap = kPanelBins;  // longest panel that converged of late
  float cb = 0.0f;  // carrier slope
  double Rr = 1.0, Ri = 0.0;  // e^{32 i b}
  PS.E[lane] = make_double2(1.0, 0.0);
  while (i < i1) {
    // modes whose next knot lies at or before bin i move on
    unsigned move = __ballot_sync(0xffffffffu, mine && k < L - 1 && next <= i);
    while (move) {
      cap = min(2 * cap, kPanelBins);
      const bool go = (move >> lane) & 1u;
      for (unsigned t = move; t; t &= t - 1) {
        const int m = __ffs(t) - 1;
        const int left = __shfl_sync(0xffffffffu, k, m);
        const int last = __shfl_sync(0xffffffffu, klast, m);
        if (left >= 0 && left + kPanelRing <= last) fetch(m, left + kPanelRing);
      }
      copy_commit();
      copy_wait<2>();  // the segment entered was asked for at least three groups ago
      __syncwarp();
      if (go) {
        ++k;
        enter();
      }
      // the segment just entered has been read before the next round's copies may take its slot
      __syncwarp();
      move = __ballot_sync(0xffffffffu, go && k < L - 1 && next <= i);
    }
    __syncwarp();
    // bins up to the next knot of any mode; the modes' phase slopes (rad per bin) at both ends
    int e = __reduce_min_sync(0xffffffffu, (mine && k < L - 1) ? next : i1);
    e = min(min(e, i1), i + cap);
    int n = e - i;
    const unsigned act = __ballot_sync(0xffffffffu, gate != 2);
    if (act == 0u) {
      if (GH) panel_direct<1, false, GH>(A, gh, PS, b, i, n, lane, k0, df, dr, di, hh);  // h = 0
      i = e;
      continue;
    }
    if (__any_sync(0xffffffffu, gate == 0)) {
      panel_direct<1, true, GH>(A, gh, PS, b, i, n, lane, k0, df, dr, di, hh);
      i = e;
      continue;
    }
    float mx = -INFINITY, mn = INFINITY, cv = 0.0f;
    if (gate != 2) {
      const float4 a = PS.sl[lane];
      const float ta = (float)((double)i - PS.kb[lane]), tz = ta + (float)(n - 1);
      const float sa = fmaf(fmaf(a.z, ta, a.y), ta, a.x), sz = fmaf(fmaf(a.z, tz, a.y), tz, a.x);
      mx = fmaxf(sa, sz);
      mn = fminf(sa, sz);
      cv = mx - mn;
    }
    mx = order_value(__reduce_max_sync(0xffffffffu, order_key(mx)));
    mn = order_value(__reduce_min_sync(0xffffffffu, order_key(mn)));
    cv = order_value(__reduce_max_sync(0xffffffffu, order_key(cv)));
    // residual phase of the panel with a centred carrier: linear 0.25 (mx - mn) n, quadratic
    // cv n / 8 (a slope change of cv over n bins), both shrinking with n
    const float lin = 0.25f * (mx - mn) * n, quad = 0.125f * cv * n;
    if (lin > kPanelDelta || quad > kPanelQuad) {
      const float fit = n * fminf(1.0f, fminf(kPanelDelta / lin, sqrtf(kPanelQuad / quad)));
      if (!(fit >= (float)kPanelMinBins)) {
        n = min(n, kPanelDirect);
        panel_direct<2, false, GH>(A, gh, PS, b, i, n, lane, k0, df, dr, di, hh);
        i += n;
        continue;
      }
      const int pieces = (int)ceilf((float)n / fit);
      n = min((n + pieces - 1) / pieces, (int)fit);
    }
    if (!(0.5f * fmaxf(fabsf(mx - cb), fabsf(mn - cb)) * n <= kPanelDelta)) {
      cb = 0.5f * (mx + mn);
      double er, ei;
      sincos_cw((double)cb * (double)lane, &ei, &er);
      PS.E[lane] = make_double2(er, ei);
      sincos_cw(32.0 * (double)cb, &Ri, &Rr);
    }
    double center, half;
    bool smooth;
    for (;;) {
      center = 0.5 * (double)(n - 1);
      half = fmax(center, 0.5);
      panel_nodes(PS, M, lane, k0 + (double)i, center, half, df, (double)cb);
      smooth = panel_smooth(PS, lane);
      if (smooth || n <= kPanelMinBins) break;
      n >>= 1;
      cap = n;
    }
    if (!smooth) {
      panel_direct<2, false, GH>(A, gh, PS, b, i, n, lane, k0, df, dr, di, hh);
      i += n;
      continue;
    }
    if constexpr (GH) {
      panel_bins_gh(A, gh, PS, i, n, center, 1.0 / half, lane, Rr, Ri, dr, di, hh);
    } else {
      double zr, zi;
      panel_bins(A, PS, i, n, center, 1.0 / half, lane, Rr, Ri, zr, zi, hh);
      const double2 E = PS.E[lane];
      dr = fma(zr, E.x, fma(-zi, E.y, dr));
      di -= fma(zr, E.y, zi * E.x);
    }
    i += n;
  }
  copy_wait<0>();
  __syncwarp();
}

}  // namespace bbhx
