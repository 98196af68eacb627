// Adjoint of the TDI response at one point (reverse of response_point, response_model.cuh).
//
// A gradient needs, of each point's transfer functions T_c, only the real number
// dL = Re(sum_c u_c dT_c) for weights u_c that are known before the point is visited.  The response
// depends on the source's angles through nine symmetric complex numbers H (linearly) and the vector
// k of its (binary, mode), on the time t = t(f) + t_ref and on f, so one reverse sweep in plain
// FP64 gives d L / d (H, k, t, f) of the point; the sums over the points of d L / d H and d L / d k
// are contracted with d (H, k) / d (phi_ref, inc, psi, lam, beta) once per (binary, mode).
// Carrying the angles' tangents through every point instead took four sweeps of the whole model
// with three tangents each.
#pragma once

#include "response_model.cuh"

namespace bbhx {

// TDI combinations of the single-link responses (Response.cu:197-261) as a table: channel c is
// factor_c (tdi_factors) times the sum of (p + q z) G over the link responses G, z = e^{2ix}.
// Links in the order (G12, G21), (G23, G32), (G31, G13).
struct TdiWeight {
  double p, q;
};
__constant__ TdiWeight kTdi[2][3][2][3] = {
    // X = G21 + z G12 - G31 - z G13, Y = G32 + z G23 - G12 - z G21, Z = G13 + z G31 - G23 - z G32
    {{{{0, 1}, {-1, 0}, {0, 0}}, {{1, 0}, {0, -1}, {0, 0}}},
     {{{0, 0}, {0, 1}, {-1, 0}}, {{0, 0}, {1, 0}, {0, -1}}},
     {{{-1, 0}, {0, 0}, {0, 1}}, {{0, -1}, {0, 0}, {1, 0}}}},
    // A: (1 + z)(G31 + G13) - G23 - z G32 - G21 - z G12,
    // E: (1 - z)(G13 - G31) + (2 + z)(G12 - G32) + (1 + 2 z)(G21 - G23),
    // T: G21 - G12 + G32 - G23 + G13 - G31
    {{{{0, -1}, {2, 1}, {-1, 0}}, {{-1, 0}, {1, 2}, {1, 0}}},
     {{{-1, 0}, {-1, -2}, {-1, 0}}, {{0, -1}, {-2, -1}, {1, 0}}},
     {{{1, 1}, {-1, 1}, {-1, 0}}, {{1, 1}, {1, -1}, {1, 0}}}}};

// H and k of one (binary, mode), the symmetric H as xx, yy, zz, xy, xz, yz
struct ResponseVec {
  double re[6], im[6], k[3];
};
__device__ __forceinline__ int sym_index(int i) { return i < 3 ? 4 * i : (i < 5 ? i - 2 : 5); }  // in H[9]

// s = sin(x y) / y for one side y = 1 -+ kn of a link and ds = d s / d y, given inv = 1 / y and the
// sine and cosine of x y; by series where those cancel (a source along the link).
__device__ __forceinline__ void sinc_side(double x, double y, double inv, double sn, double cs,
                                          double* s, double* ds) {
  if (y > 1e-3) {
    *s = sn * inv;
    *ds = (x * cs - *s) * inv;
    return;
  }
  const double w = x * y, w2 = w * w;
  *s = x * (1.0 - w2 * (1.0 / 6.0 - w2 * (1.0 / 120.0)));
  *ds = -x * x * w * (1.0 / 3.0 - w2 * (1.0 / 30.0 - w2 * (1.0 / 840.0)));
}

// Value and time derivative of the 3-vector at `offset` of the orbit table (orbit_lerp).
struct OrbitVec {
  V3T<double> v, d;
};
__device__ __forceinline__ OrbitVec orbit_vec(const double* lo, int stride, int offset, double frac,
                                              double inv_dt) {
  if (lo == nullptr) return OrbitVec{{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
  lo += offset;
  const double* hi = lo + stride;
  const double x = __ldg(lo), y = __ldg(lo + 1), z = __ldg(lo + 2);
  const double dx = __ldg(hi) - x, dy = __ldg(hi + 1) - y, dz = __ldg(hi + 2) - z;
  return OrbitVec{{x + dx * frac, y + dy * frac, z + dz * frac},
                  {dx * inv_dt, dy * inv_dt, dz * inv_dt}};
}

// The links' part: adds d L / d (H, k) of dL = Re(sum_c u_c dT_c) to `a`, d L / d t to *tbar and,
// WITH_F, d L / d f to *fbar; returns sum_c u_c T_c.  r is the (binary, mode)'s own H and k.
template <bool WITH_F>
__device__ __forceinline__ cplx links_adjoint(const ResponseVec& r, const OrbitTables& orb,
                                              double f, double t, const cplx (&u)[3], int TDItag,
                                              int rescaled, int tdi2, ResponseVec& a, double* tbar,
                                              double* fbar) {
  const double x = f * orb.pi_L_over_c;
  cplx cb[3], cbx[3];  // u_c factor_c and its d / dx
  cplx e1;
  if constexpr (WITH_F) {
    using D = ad::Dual<1>;
    D xd(x);
    xd.d[0] = 1.0;
    const cplxT<D> e1d = expi(xd);
    cplxT<D> fac[3];
    tdi_factors(e1d, TDItag, rescaled, tdi2, fac);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      cb[c] = u[c] * cmk(fac[c].re.v, fac[c].im.v);
      cbx[c] = u[c] * cmk(fac[c].re.d[0], fac[c].im.d[0]);
    }
    e1 = cmk(e1d.re.v, e1d.im.v);
  } else {
    e1 = expi(x);
    tdi_factors(e1, TDItag, rescaled, tdi2, cb);
#pragma unroll
    for (int c = 0; c < 3; ++c) cb[c] = u[c] * cb[c];
  }
  const cplx z = e1 * e1;
  const OrbitWindow<double> win = orbit_window(orb, t);
  const TdiWeight(*tdi)[2][3] = kTdi[TDItag == 1 ? 0 : 1];
  const double xL = x * orb.inv_armlength;
  cplx ut = cmk(0.0, 0.0);
  double xbar = 0.0, tb = 0.0;
  // not unrolled: three copies of the body are longer than the instruction cache serves well
#pragma unroll 1
  for (int l = 0; l < 3; ++l) {
    const OrbitVec n = orbit_vec(win.n_lo, 18, orb.link_index[l == 0 ? 2 : l - 1] * 3, win.frac,
                                 orb.inv_dt);
    OrbitVec p = orbit_vec(win.x_lo, 9, 3 * l, win.frac, orb.inv_dt);
    {
      const OrbitVec q = orbit_vec(win.x_lo, 9, l == 2 ? 0 : 3 * (l + 1), win.frac, orb.inv_dt);
      p.v.x += q.v.x, p.v.y += q.v.y, p.v.z += q.v.z;
      p.d.x += q.d.x, p.d.y += q.d.y, p.d.z += q.d.z;
    }
    const double kn = r.k[0] * n.v.x + r.k[1] * n.v.y + r.k[2] * n.v.z;
    const double kp = r.k[0] * p.v.x + r.k[1] * p.v.y + r.k[2] * p.v.z;
    const double w = 1.0 + kp * orb.inv_armlength;
    // H n, and h = n H n
    const double ar = r.re[0] * n.v.x + r.re[3] * n.v.y + r.re[4] * n.v.z;
    const double br = r.re[3] * n.v.x + r.re[1] * n.v.y + r.re[5] * n.v.z;
    const double cr = r.re[4] * n.v.x + r.re[5] * n.v.y + r.re[2] * n.v.z;
    const double ai = r.im[0] * n.v.x + r.im[3] * n.v.y + r.im[4] * n.v.z;
    const double bi = r.im[3] * n.v.x + r.im[1] * n.v.y + r.im[5] * n.v.z;
    const double ci = r.im[4] * n.v.x + r.im[5] * n.v.y + r.im[2] * n.v.z;
    const cplx h = cmk(ar * n.v.x + br * n.v.y + cr * n.v.z, ai * n.v.x + bi * n.v.y + ci * n.v.z);
    const cplx e = expi(x * w);
    // the two directions' x sinc(x (1 -+ kn)): sines and cosines by the addition theorems
    double sk, ck;
    model_sincos(x * kn, &sk, &ck);
    // 1 / (1 -+ kn) by one division of 1 - kn^2, which cancels for a source along the link
    const double ym = 1.0 - kn, yp = 1.0 + kn, den = 1.0 - kn * kn;
    double im = 1.0 / den, ip = im;
    if (den > 1e-3) {
      im *= yp;
      ip *= ym;
    } else {
      im = 1.0 / ym;
      ip = 1.0 / yp;
    }
    const double cm = e1.re * ck + e1.im * sk, cp = e1.re * ck - e1.im * sk;
    double sm, dsm, sp, dsp;
    sinc_side(x, ym, im, e1.im * ck - e1.re * sk, cm, &sm, &dsm);
    sinc_side(x, yp, ip, e1.im * ck + e1.re * sk, cp, &sp, &dsp);
    // weights of the two directions' G = s i h e
    cplx wm = cmk(0.0, 0.0), wp = cmk(0.0, 0.0);
    cplx xm = cmk(0.0, 0.0), xp = cmk(0.0, 0.0);  // d / dx of the weights
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const TdiWeight g0 = tdi[l][0][c], g1 = tdi[l][1][c];
      const cplx z0 = cmk(g0.p + g0.q * z.re, g0.q * z.im), z1 = cmk(g1.p + g1.q * z.re, g1.q * z.im);
      wm = wm + cb[c] * z0;
      wp = wp + cb[c] * z1;
      if constexpr (WITH_F) {  // dz / dx = 2 i z
        xm = xm + cbx[c] * z0 + (2.0 * g0.q) * (cb[c] * times_i(z));
        xp = xp + cbx[c] * z1 + (2.0 * g1.q) * (cb[c] * times_i(z));
      }
    }
    const cplx ie = times_i(e), ihe = h * ie;
    const cplx q = (sm * wm + sp * wp) * ie;  // dL = Re(q dh)
    const cplx qh = q * h;
    ut = ut + qh;
    const double gm = wm.re * ihe.re - wm.im * ihe.im, gp = wp.re * ihe.re - wp.im * ihe.im;
    const double knb = gp * dsp - gm * dsm;   // dL / d (k.n): y = 1 -+ kn
    const double kpb = -qh.im * xL;           // dL / d (k.p)
    const double nx = n.v.x, ny = n.v.y, nz = n.v.z;
    const double m6[6] = {nx * nx, ny * ny, nz * nz, 2.0 * nx * ny, 2.0 * nx * nz, 2.0 * ny * nz};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      a.re[i] += q.re * m6[i];
      a.im[i] -= q.im * m6[i];
    }
    a.k[0] += knb * nx + kpb * p.v.x;
    a.k[1] += knb * ny + kpb * p.v.y;
    a.k[2] += knb * nz + kpb * p.v.z;
    const double q2r = 2.0 * q.re, q2i = 2.0 * q.im;
    tb += (knb * r.k[0] + q2r * ar - q2i * ai) * n.d.x +
          (knb * r.k[1] + q2r * br - q2i * bi) * n.d.y +
          (knb * r.k[2] + q2r * cr - q2i * ci) * n.d.z +
          kpb * (r.k[0] * p.d.x + r.k[1] * p.d.y + r.k[2] * p.d.z);
    if constexpr (WITH_F) {
      const cplx xs = sm * xm + sp * xp;
      xbar += gm * cm + gp * cp - qh.im * w + (xs.re * ihe.re - xs.im * ihe.im);
    }
  }
  *tbar += tb;
  if constexpr (WITH_F) *fbar += xbar * orb.pi_L_over_c;
  return ut;
}

// Roemer delay R = 2 pi f k.(AU (cos al, sin al, 0)) / c at al = Omega0 t
struct RoemerPoint {
  double sa, ca, sc;  // sc = 2 pi f AU / c
};
__device__ __forceinline__ double roemer(const ResponseVec& r, double f, double t, RoemerPoint* p) {
  model_sincos(Omega0 * t, &p->sa, &p->ca);
  p->sc = 2. * PI / C_SI * f * AU_SI;
  return p->sc * (r.k[0] * p->ca + r.k[1] * p->sa);
}
// adds its adjoint, dL = phibar dR (f apart: R / f)
__device__ __forceinline__ void roemer_adjoint(const ResponseVec& r, const RoemerPoint& p,
                                               double phibar, ResponseVec& a, double* tbar) {
  const double w = phibar * p.sc;
  a.k[0] += w * p.ca;
  a.k[1] += w * p.sa;
  *tbar += w * Omega0 * (r.k[1] * p.ca - r.k[0] * p.sa);
}

}  // namespace bbhx
