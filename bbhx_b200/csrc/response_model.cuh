// Fast frequency-domain LISA TDI response (device side).
//
// Follows the reference's response (src/bbhx/cutils/Response.cu), i.e. the
// Marsat & Baker fast FD response (arXiv:1806.10734, 2003.00357):
//   * per (binary, mode): wave vector k, polarisation tensors H+ / Hx rotated into the
//     SSB frame, and the complex mode matrix H = Y+ H+ + Yx Hx from the spin-weighted
//     spherical harmonics (Response.cu:468-608);
//   * per (binary, mode, frequency): single-link transfer functions G_slr at the
//     spacecraft positions for time t = t(f) (Response.cu:54-194), combined into
//     XYZ or AET (optionally 2nd-generation) TDI (Response.cu:197-261), plus the
//     orbital Roemer delay 2 pi f k.R / c added to the phase (Response.cu:264-314).
// The per-(binary, mode) part is computed once (ResponseMode) instead of by thread 0 of
// every block; the orbit tables are read through the __ldg path.
//
// Orbit tables (bbhx_b200/orbits.py): x_arr[N][3][3], n_arr[N][6][3], link order
// links[6]; sample k at t = k dt; linear interpolation for 0 <= floor(t/dt) < N-1, zero
// vector outside.  The window and its fraction are found once per time and shared by the six
// vectors read there.
#pragma once

#include "bbhx_common.cuh"
#include "dual.cuh"

namespace bbhx {

struct OrbitTables {
  const double* x_arr;  // [N][3][3]
  const double* n_arr;  // [N][6][3]
  double dt;
  double inv_dt;  // 1 / dt
  int N;
  int link_index[3];  // table slots of links 12, 23, 31
  double armlength;
  double inv_armlength;  // 1 / armlength
  double pi_L_over_c;    // pi armlength / c
};

// Device-resident orbit tables owned by the C-ABI orbit handle (bbhx_orbits_*).
struct OrbitHandle {
  double* d_x = nullptr;
  double* d_n = nullptr;
  OrbitTables tab{};
  bool ready = false;
};

template <typename T>
struct ResponseModeT {
  cplxT<T> H[9];  // complex mode matrix, row-major
  T k[3];         // propagation direction
};
using ResponseMode = ResponseModeT<double>;


template <typename T>
struct V3T {
  T x, y, z;
};

// Table window of time t: w = floor(t / dt) (the lookup rule), valid for 0 <= w < N - 1, and the
// interpolation fraction (t - w dt) / dt shared by all vectors read at that time.
template <typename T>
struct OrbitWindow {
  const double* x_lo;  // first x row of the window (nullptr when outside the table)
  const double* n_lo;
  T frac;
};

template <typename T>
__device__ __forceinline__ OrbitWindow<T> orbit_window(const OrbitTables& orb, const T& t) {
  OrbitWindow<T> w;
  const double f = floor(value_of(t) / orb.dt);
  if (!(f >= 0.0) || f >= (double)(orb.N - 1)) {
    w.x_lo = nullptr;
    w.n_lo = nullptr;
    w.frac = T(0.0);
    return w;
  }
  const int wi = (int)f;
  w.x_lo = orb.x_arr + (size_t)wi * 9;
  w.n_lo = orb.n_arr + (size_t)wi * 18;
  w.frac = (t - wi * orb.dt) * orb.inv_dt;
  return w;
}

// lo + (hi - lo) * frac of the 3-vector at `offset` of rows lo and lo + stride; zero vector
// outside the table.
template <typename T>
__device__ __forceinline__ V3T<T> orbit_lerp(const double* lo, int stride, int offset,
                                             const T& frac) {
  if (lo == nullptr) return V3T<T>{T(0.0), T(0.0), T(0.0)};
  lo += offset;
  const double* hi = lo + stride;
  V3T<T> r;
  r.x = __ldg(lo + 0) + (__ldg(hi + 0) - __ldg(lo + 0)) * frac;
  r.y = __ldg(lo + 1) + (__ldg(hi + 1) - __ldg(lo + 1)) * frac;
  r.z = __ldg(lo + 2) + (__ldg(hi + 2) - __ldg(lo + 2)) * frac;
  return r;
}
// spin-weight -2 spherical harmonics for l = 2..4 (Response.cu:383-424)
template <typename T>
__device__ inline cplxT<T> sylm_m2(int l, int m, const T& theta, const T& phi) {
  T fac = 0.0;
  T ct = cos(theta), st = sin(theta);
  T c2 = cos(theta / 2.0), s2 = sin(theta / 2.0);
  if (l == 2) {
    if (m == -2) fac = sqrt(5.0 / (64.0 * PI)) * (1.0 - ct) * (1.0 - ct);
    else if (m == -1) fac = sqrt(5.0 / (16.0 * PI)) * st * (1.0 - ct);
    else if (m == 1) fac = sqrt(5.0 / (16.0 * PI)) * st * (1.0 + ct);
    else if (m == 2) fac = sqrt(5.0 / (64.0 * PI)) * (1.0 + ct) * (1.0 + ct);
  } else if (l == 3) {
    if (m == -3) fac = sqrt(21.0 / (2.0 * PI)) * c2 * pow(s2, 5.0);
    else if (m == -2) fac = sqrt(7.0 / (4.0 * PI)) * (2.0 + 3.0 * ct) * pow(s2, 4.0);
    else if (m == 2) fac = sqrt(7.0 / PI) * pow(c2, 4.0) * (-2.0 + 3.0 * ct) / 2.0;
    else if (m == 3) fac = -sqrt(21.0 / (2.0 * PI)) * pow(c2, 5.0) * s2;
  } else if (l == 4) {
    if (m == -4) fac = 3.0 * sqrt(7.0 / PI) * pow(c2, 2.0) * pow(s2, 6.0);
    else if (m == -3) fac = 3.0 * sqrt(7.0 / (2.0 * PI)) * c2 * (1.0 + 2.0 * ct) * pow(s2, 5.0);
    else if (m == 3) fac = -3.0 * sqrt(7.0 / (2.0 * PI)) * pow(c2, 5.0) * (-1.0 + 2.0 * ct) * s2;
    else if (m == 4) fac = 3.0 * sqrt(7.0 / PI) * pow(c2, 6.0) * pow(s2, 2.0);
  }
  if (m == 0) return cmk(fac, T(0.0));
  T s, c;
  sincos(m * phi, &s, &c);
  return cmk(fac * c, fac * s);
}

template <typename T>
__device__ inline void response_mode_setup(ResponseModeT<T>& r, int ell, int mm, const T& phi_ref,
                                           const T& inc, const T& lam, const T& beta,
                                           const T& psi) {
  T cl = cos(lam), sl = sin(lam), cb = cos(beta), sb = sin(beta), cp = cos(psi), sp = sin(psi);
  r.k[0] = -cb * cl;
  r.k[1] = -cb * sl;
  r.k[2] = -sb;
  // rotation from the wave frame to the SSB frame and its inverse
  T O[9] = {cp * sl - cl * sb * sp, -cl * cp * sb - sl * sp, -cb * cl,
            -cl * cp - sb * sl * sp, -cp * sb * sl + cl * sp, -cb * sl,
            cb * sp, cb * cp, -sb};
  T Oi[9] = {O[0], O[3], O[6], O[1], O[4], O[7], O[2], O[5], O[8]};
  // H+ = O diag(1,-1,0) O^-1, Hx = O offdiag(1,1) O^-1
  T Hp[9], Hc[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      // (HS+ O^-1)_{kj} = s_k Oi[k][j] with s = (1,-1,0); (HSx O^-1)_{0j} = Oi[1][j], _{1j} = Oi[0][j]
      T p = O[i * 3 + 0] * Oi[0 * 3 + j] - O[i * 3 + 1] * Oi[1 * 3 + j];
      T x = O[i * 3 + 0] * Oi[1 * 3 + j] + O[i * 3 + 1] * Oi[0 * 3 + j];
      Hp[i * 3 + j] = p;
      Hc[i * 3 + j] = x;
    }
  cplxT<T> Ylm = sylm_m2(ell, mm, inc, phi_ref);
  cplxT<T> Ylmm = sylm_m2(ell, -mm, inc, phi_ref);
  double sgn = (ell % 2 == 0) ? 1.0 : -1.0;
  cplxT<T> Yl_m = sgn * conj(Ylmm);
  cplxT<T> Yp = 0.5 * (Ylm + Yl_m);
  cplxT<T> Yc = times_i(0.5 * (Ylm - Yl_m));
  for (int q = 0; q < 9; ++q) r.H[q] = Yp * Hp[q] + Yc * Hc[q];
}

template <typename T>
struct TransferT {
  cplxT<T> L1, L2, L3;
  T phaseRdelay;
};
using Transfer = TransferT<double>;

// n H n of the symmetric mode matrix
template <typename T>
__device__ __forceinline__ cplxT<T> nHn(const cplxT<T>* H, const V3T<T>& n) {
  const T xy = 2.0 * n.x * n.y, xz = 2.0 * n.x * n.z, yz = 2.0 * n.y * n.z;
  const T xx = n.x * n.x, yy = n.y * n.y, zz = n.z * n.z;
  return cmk(H[0].re * xx + H[4].re * yy + H[8].re * zz + H[1].re * xy + H[2].re * xz + H[5].re * yz,
             H[0].im * xx + H[4].im * yy + H[8].im * zz + H[1].im * xy + H[2].im * xz + H[5].im * yz);
}

template <typename T>
__device__ __forceinline__ T sinc(const T& x) { return x == 0.0 ? T(1.0) : sin(x) / x; }

// x sinc(x (1 - kn)) and x sinc(x (1 + kn)) from (s1, c1) = sin, cos of x: the sines by the
// addition theorem from one sine / cosine of x kn, the two divisions by one of 1 - kn^2 (a source
// along the link, 1 - kn^2 -> 0, takes the plain form).
template <typename T>
__device__ __forceinline__ void sinc_pair(const T& x, const T& s1, const T& c1, const T& kn, T* minus,
                                          T* plus) {
  const T den = 1.0 - kn * kn;
  if (!(den > 1e-6)) {
    *minus = x * sinc(x * (1.0 - kn));
    *plus = x * sinc(x * (1.0 + kn));
    return;
  }
  T sk, ck;
  model_sincos(x * kn, &sk, &ck);
  const T inv = 1.0 / den, a = s1 * ck, b = c1 * sk;
  *minus = (a - b) * ((1.0 + kn) * inv);
  *plus = (a + b) * ((1.0 - kn) * inv);
}

// Frequency factors of the three TDI channels (Response.cu:197-261), e1 = e^{ix}: X, Y, Z share
// one; A, E, T carry their normalisations.
template <typename T>
__device__ __forceinline__ void tdi_factors(const cplxT<T>& e1, int TDItag, int rescaled, int tdi2,
                                            cplxT<T> (&fac)[3]) {
  const cplxT<T> one = cmk(T(1.0), T(0.0)), z = e1 * e1;
  const T s2x = 2. * e1.im * e1.re;
  if (TDItag == 1) {
    fac[0] = fac[1] = fac[2] = rescaled ? one : times_i(2. * s2x * z);
    return;
  }
  cplxT<T> fAE = one, fT = one;
  if (!rescaled) {
    fAE = times_i(SQRT2 * s2x * z);
    fT = (2. * SQRT2 * s2x * e1.im) * (z * e1);
  }
  if (tdi2) {
    const cplxT<T> f2 = times_i((-2. * (2. * s2x * z.re)) * (z * z));  // -2i sin4x e^{4ix}
    fAE = f2 * fAE;
    fT = f2 * fT;
  }
  fac[0] = fAE;
  fac[1] = INVSQRT3 * fAE;
  fac[2] = (2. * INVSQRT6) * fT;
}

// TDItag: 1 = XYZ, 2 = AET.  f in Hz, t in s.  The frequency has its own type F: double, or
// the dual type T when the frequency itself carries tangents (knots that move with theta).
template <typename T, typename F = double>
__device__ inline TransferT<T> response_point(const ResponseModeT<T>& r, const OrbitTables& orb,
                                              const F& f, const T& t, int TDItag, int rescaled,
                                              int tdi2) {
  const T* k = r.k;
  // Roemer delay relative to the SSB (circular 1 AU orbit of the guiding centre)
  T al = Omega0 * t;
  T sa, ca;
  model_sincos(al, &sa, &ca);
  T kR = AU_SI * (k[0] * ca + k[1] * sa);
  TransferT<T> out;
  out.phaseRdelay = 2. * PI / C_SI * f * kR;

  const OrbitWindow<T> win = orbit_window(orb, t);
  V3T<T> p1 = orbit_lerp(win.x_lo, 9, 0, win.frac);
  V3T<T> p2 = orbit_lerp(win.x_lo, 9, 3, win.frac);
  V3T<T> p3 = orbit_lerp(win.x_lo, 9, 6, win.frac);
  V3T<T> n1 = orbit_lerp(win.n_lo, 18, orb.link_index[0] * 3, win.frac);
  V3T<T> n2 = orbit_lerp(win.n_lo, 18, orb.link_index[1] * 3, win.frac);
  V3T<T> n3 = orbit_lerp(win.n_lo, 18, orb.link_index[2] * 3, win.frac);
  T kn1 = k[0] * n1.x + k[1] * n1.y + k[2] * n1.z;
  T kn2 = k[0] * n2.x + k[1] * n2.y + k[2] * n2.z;
  T kn3 = k[0] * n3.x + k[1] * n3.y + k[2] * n3.z;
  cplxT<T> n1H = nHn(r.H, n1), n2H = nHn(r.H, n2), n3H = nHn(r.H, n3);
  const double invL = orb.inv_armlength;
  const T kp1 = k[0] * p1.x + k[1] * p1.y + k[2] * p1.z;
  const T kp2 = k[0] * p2.x + k[1] * p2.y + k[2] * p2.z;
  const T kp3 = k[0] * p3.x + k[1] * p3.y + k[2] * p3.z;
  T pre = f * orb.pi_L_over_c;
  cplxT<T> e12 = expi(pre * (1. + (kp1 + kp2) * invL));
  cplxT<T> e23 = expi(pre * (1. + (kp2 + kp3) * invL));
  cplxT<T> e31 = expi(pre * (1. + (kp3 + kp1) * invL));
  // e^{ix}, x = pre, and its powers / sines from one sincos
  const cplxT<T> e1 = expi(pre);
  const cplxT<T> z = e1 * e1;  // e^{2ix}
  // The constellation-centre phase factor exp(+i 2 pi f k.p0 / c) of the full response and
  // the Roemer-delay factor exp(-i phaseRdelay) cancel identically (Response.cu:166,304-309).
  const cplxT<T> c3 = times_i(n3H * e12), c1 = times_i(n1H * e23), c2 = times_i(n2H * e31);
  T sm, sp;
  sinc_pair(pre, e1.im, e1.re, kn3, &sm, &sp);
  const cplxT<T> G12 = sm * c3, G21 = sp * c3;
  sinc_pair(pre, e1.im, e1.re, kn1, &sm, &sp);
  const cplxT<T> G23 = sm * c1, G32 = sp * c1;
  sinc_pair(pre, e1.im, e1.re, kn2, &sm, &sp);
  const cplxT<T> G31 = sm * c2, G13 = sp * c2;
  cplxT<T> fac[3];
  tdi_factors(e1, TDItag, rescaled, tdi2, fac);
  if (TDItag == 1) {
    out.L1 = fac[0] * (G21 + z * G12 - G31 - z * G13);
    out.L2 = fac[1] * (G32 + z * G23 - G12 - z * G21);
    out.L3 = fac[2] * (G13 + z * G31 - G23 - z * G32);
    return out;
  }
  const cplxT<T> one = cmk(T(1.0), T(0.0));
  out.L1 = fac[0] * ((one + z) * (G31 + G13) - G23 - z * G32 - G21 - z * G12);
  out.L2 = fac[1] * ((one - z) * (G13 - G31) + (cmk(T(2.0), T(0.0)) + z) * (G12 - G32) +
                     (one + 2. * z) * (G21 - G23));
  out.L3 = fac[2] * (G21 - G12 + G32 - G23 + G13 - G31);
  return out;
}

}  // namespace bbhx
