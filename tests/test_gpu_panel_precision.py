"""<d|h> and <h|h> of the FP64 panels (csrc/direct_panel.cuh) against 80-bit sums of the library's
own spline sets: x87 extended arithmetic keeps a phase of 1e7 rad to 5e-13 rad, so the comparison
sees what the panels round and truncate, which a bin-by-bin FP64 evaluation (4e-10 to 9e-9) cannot
show.  Wide spline segments beside a zero of the TDI response, where the phase moves by 4e5 rad
within a segment and <h|h> comes from a few hundred bins; an ordinary band; grids of 24, 33 and 129
bins.  Each source alone (items of 256 bins), in a batch (items of 8192 where the grid is that long),
and through the gradient's kernel.

Tolerance: the panels stop at degree 7, and the convergence check admits coefficients c_6, c_7 up to
1.6e-8 of the largest.  The next one is then below 0.15 / 8 of that (the residual phase is 0.15 rad
over a half panel), 3e-10, and its Chebyshev remainder 2^-7 of it, 2.3e-12 of the largest |h| of the
panel; the nodes' rounding (1e-15) is far inside.  With H_i the largest |h| within 1024 bins (a
panel's length) and E = 2.5e-12, each bin may be off by E H_i, all the same way; the FP64 sums add
1e-13 of sqrt(<d|d> <h|h>) and <h|h>."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

YEAR = 31558149.763545603
E = 2.5e-12
# m1, m2 [Msun], chi1z, chi2z, phi_ref, inc, lam, beta, psi, t_ref / observation time
SOURCES = [(1.95394e5, 7.2803e4, -0.0526, -0.3700, 2.9403, 2.2184, 0.4744, 0.9369, 2.3605, 0.8828),
           (1.59500e5, 1.39473e5, -0.1683, 0.7664, 4.2924, 1.5793, 0.4417, -0.5580, 1.6414, 0.9065),
           (2.54432e5, 5.4472e4, 0.7199, 0.2592, 2.9846, 1.6356, 3.4849, -0.4804, 2.6761, 0.8314)]


def _params(tobs):
    s = np.array(SOURCES).T
    return np.array([*s[:4], np.full(3, 2e27), s[4], np.zeros(3), *s[5:9], s[9] * tobs * YEAR])


def _exact_grid(f):
    """k0 and df of the kernels' record: the first of their candidates that gives every f = k df."""
    n = len(f)
    k0 = np.rint(f[0] / ((f[-1] - f[0]) / (n - 1)))
    df = f[-1] / (k0 + n - 1)
    for c in (df, np.nextafter(df, 0.0), np.nextafter(df, 1.0)):
        if np.array_equal((k0 + np.arange(n)) * c, f):
            return k0, c
    raise AssertionError("not a uniform grid")


def _template(f, x, q, ts, te):
    """h [3, N] in 80 bits of one binary: knots x [M, L], q [4, 9, M, L] = y, c1, c2, c3."""
    ld = np.longdouble
    k0, df = _exact_grid(f)
    k = (ld(k0) + np.arange(len(f)).astype(ld)) * ld(df)
    h = np.zeros((3, len(f)), np.clongdouble)
    for m in range(x.shape[0]):
        s = np.searchsorted(x[m], f, side="right") - 1
        ok = (s >= 0) & (s < x.shape[1] - 1)
        s = np.where(ok, s, 0)
        u = k - x[m][s].astype(ld)
        v = [((q[3, p, m, s].astype(ld) * u + q[2, p, m, s]) * u + q[1, p, m, s]) * u + q[0, p, m, s]
             for p in range(9)]
        amp = np.where(ok & (v[2] >= ts) & ((v[2] <= te) | (te <= 0.0)), v[0], ld(0))
        c, s = amp * np.cos(v[1]), amp * np.sin(v[1])
        for ch in range(3):
            tr, ti = v[3 + 2 * ch], v[4 + 2 * ch]
            h[ch] += (tr * c - ti * s) - 1j * (tr * s + ti * c)
    return h


def _largest_near(h, reach=1024):
    a = np.pad(np.abs(h).astype(np.float64), ((0, 0), (reach, reach)))
    return np.lib.stride_tricks.sliding_window_view(a, 2 * reach + 1, axis=1).max(axis=2)


@pytest.mark.parametrize("tobs,lo,bins,length,modes,batch", [
    (1.0, 0.0592, 44000, 256, None, 2400),
    (0.5, 0.0592, 22000, 256, None, 33),
    (0.8, 0.0592, 35000, 382, [(2, 2), (3, 3), (4, 4)], 6),
    (0.3, 0.0200, 14000, 1000, None, 30),
    (0.1, 0.0500, 24, 600, None, 3),
    (0.1, 0.0500, 33, 600, None, 3),
    (0.1, 0.0500, 129, 600, None, 3),
])
def test_sums_against_80_bits(tobs, lo, bins, length, modes, batch):
    import torch

    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits, Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import gaussian_noise, notch_tdi_zeros

    assert np.finfo(np.longdouble).nmant >= 63
    df = 1.0 / (tobs * YEAR)
    f = (math.ceil(lo / df) + np.arange(bins)) * df
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))
    like = Likelihood(wave, f, gaussian_noise(psd, df, 5), psd)
    P = _params(tobs)
    kw = dict(length=length, modes=modes, t_obs_start=0.0, t_obs_end=tobs)

    def sums(params):
        like.get_ll(params, **kw)
        return like.d_h.cpu().numpy(), like.h_h.cpu().numpy().real

    alone = [sums(P[:, b:b + 1]) for b in range(3)]
    many = sums(np.tile(P, (1, batch // 3)))
    grad = wave.direct_grad(torch.as_tensor(P, device="cuda"), like.data_freqs, like.data_channels,
                            like.noise_factors, **kw)
    buf, c1, c2, c3, x, ts, te = wave._spline_set(tuple(P), 0.0, tobs, length, modes)
    M = wave.num_modes
    x = x.reshape(3, M, length).cpu().numpy()
    q = np.array([a.reshape(9, 3, M, length).cpu().numpy() for a in (buf, c1, c2, c3)])
    ts, te = ts.cpu().numpy(), te.cpu().numpy()
    d = like.data_channels.reshape(3, -1).cpu().numpy()
    w = like.noise_factors.reshape(3, -1).cpu().numpy()
    for b in range(3):
        h = _template(f, x[b], q[:, :, b], ts[b], te[b])
        dh = 4 * np.sum(np.conj(d) * (w * h))
        hh = 4 * np.sum((w * h.real) ** 2 + (w * h.imag) ** 2)
        H = _largest_near(h)
        a = np.abs(h).astype(np.float64)
        tol_hh = float(8 * E * np.sum(w * w * a * H) + 1e-13 * hh)
        tol_dh = float(4 * E * np.sum(np.abs(d) * w * H) + 1e-13 * np.sqrt(like.d_d * float(hh)))
        got = [alone[b], (many[0][b::3], many[1][b::3]),
               (grad[0].cpu().numpy()[b], grad[1].cpu().numpy().real[b])]
        for name, (gd, gh) in zip(("alone", "batch", "gradient"), got):
            ed = float(np.max(np.abs(gd - np.complex128(dh))))
            eh = float(np.max(np.abs(np.atleast_1d(gh).astype(np.longdouble) - hh)))
            print(b, name, "h_h %.1e of it, allowed %.1e; d_h %.1e, allowed %.1e"
                  % (eh / float(hh), tol_hh / float(hh), ed, tol_dh))
            assert eh <= tol_hh
            assert ed <= tol_dh
