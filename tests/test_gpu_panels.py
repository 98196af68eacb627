"""The FP64 direct likelihood sums uniform grids panel by panel (csrc/direct_panel.cuh) and other
grids bin by bin.  Moving one frequency of a uniform grid by one ulp sends the same problem down
the bin-by-bin path, so the two are compared where the panel walk can go wrong: grids coarser and
finer than the knots, few knots, supports that start and end inside the grid, one mode and many,
observation windows that cut the template, item sizes on both sides of the tile rule.

Tolerance: the bin-by-bin path rounds each phase phi to FP64, at most ~8 ulp over the spline and
the reduction, so e^{i phi} is off by eps = 8 * 2^-53 * phi_max rad with phi_max = 2 pi f t; in the
worst case all bins move the same way: |d<d|h>| <= eps sqrt(<d|d> <h|h>), |d<h|h>| <= 2 eps <h|h>.
The panel sums (interpolation error 2e-13 of the template) lie far inside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

YEAR = 31558149.763545603


def _likes(tobs, lo, hi, seed):
    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits, Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import data_grid, gaussian_noise, notch_tdi_zeros

    f = data_grid(tobs, lo, hi)
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    data = gaussian_noise(psd, f[1] - f[0], seed)
    g = f.copy()
    g[len(g) // 2] = np.nextafter(g[len(g) // 2], 1.0)
    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))
    return Likelihood(wave, f, data, psd), Likelihood(wave, g, data, psd), f


@pytest.mark.parametrize("tobs,lo,hi,length,modes,batch,t_end", [
    (0.02, 1e-5, 0.1, 1024, None, 3, 1.0),          # knots closer than the bins at low frequency
    (0.1, 1e-5, 0.1, 256, [(2, 2)], 1, 1.0),        # few wide segments, one mode
    (0.3, 1e-5, 0.1, 512, None, 2, 1.0),            # the smallest item size
    (0.3, 3e-3, 4.1e-2, 333, [(3, 3), (2, 1), (4, 4)], 40, 1.0),  # ragged band, larger items
    (0.1, 2e-2, 2.1e-2, 1500, None, 5, 1.0),        # a grid of a few thousand bins
    (0.1, 1.23e-2, 1.2301e-2, 600, None, 3, 1.0),   # a few dozen bins
    (0.5, 1e-4, 0.1, 40, None, 2, 1.0),             # segments wider than a panel, steep in between
    (0.2, 1e-5, 0.1, 900, None, 4, 0.9),            # the window ends near the merger
])
def test_panels_match_bin_by_bin(tobs, lo, hi, length, modes, batch, t_end):
    from bbhx_b200.synthetic import draw_params

    uniform, nudged, f = _likes(tobs, lo, hi, 11)
    P = draw_params(batch, tobs, 17 + length)
    rng = np.random.default_rng(length)
    P[11] = rng.uniform(0.6, 0.85, batch) * tobs * YEAR
    kw = dict(length=length, modes=modes, t_obs_start=0.0, t_obs_end=tobs * t_end)
    out = []
    for like in (uniform, nudged):
        like.get_ll(P, **kw)
        out.append((like.d_h.cpu().numpy(), like.h_h.cpu().numpy().real))
    (dh, hh), (dh1, hh1) = out
    eps = 8.0 * 2.0 ** -53 * 2.0 * np.pi * f[-1] * tobs * YEAR
    print("d_h", np.max(np.abs(dh - dh1) / np.sqrt(uniform.d_d * np.maximum(hh1, 1e-300))),
          "h_h", np.max(np.abs(hh - hh1) / np.maximum(hh1, 1e-300)), "eps", eps)
    assert np.all(np.isfinite(dh)) and np.all(hh >= 0.0)
    assert np.all(np.abs(dh - dh1) <= eps * np.sqrt(uniform.d_d * hh1) + 1e-13)
    assert np.all(np.abs(hh - hh1) <= 2.0 * eps * hh1 + 1e-13)


def _interp_tdi(fd, x, y, c, ts, te, st, n):
    """Template [3, n] of one binary through InterpTDI with torch.searchsorted's segments."""
    import torch

    from bbhx_b200 import _lib

    M, L = x.shape
    seg = torch.searchsorted(x, fd[st:st + n][None].expand(M, -1).contiguous(), right=True) - 1
    inds = seg.to(torch.int32).contiguous()
    out = torch.empty((3, n), dtype=torch.complex128, device="cuda")
    one = lambda v, t: np.array([v], dtype=t)
    tp, ip = one(out.data_ptr(), np.int64), one(inds.data_ptr(), np.int64)
    a, z, i0, ln = one(float(ts), float), one(float(te), float), one(st, np.int32), one(n, np.int32)
    arrays = [v.contiguous() for v in (x, y, *c)]
    _lib.call("bbhx_InterpTDI", _lib.hptr(tp), _lib.dptr(fd), *[_lib.dptr(v) for v in arrays],
              _lib.hptr(a), _lib.hptr(z), L, len(fd), 1, M, _lib.hptr(ip), _lib.hptr(i0),
              _lib.hptr(ln), _lib.stream())
    return out


@pytest.mark.parametrize("tobs,lo,hi,length,modes,batch,nudge", [
    (0.05, 1e-5, 0.1, 1024, None, 3, False),
    (0.05, 1e-5, 0.1, 1024, None, 3, True),      # not k df: every bin searches its segment
    (0.3, 5e-4, 0.03, 300, [(2, 2)], 1, False),
    (0.1, 2e-2, 2.03e-2, 2000, [(3, 3), (4, 4)], 7, False),
    (0.1, 2e-2, 2.0001e-2, 64, [(2, 1)], 2, True),
])
def test_templates_match_bin_by_bin(tobs, lo, hi, length, modes, batch, nudge):
    """bbhx_interp_templates over whole supports against InterpTDI with given segments.
    Tolerance: both round phases of phi_max = 2 pi f t to FP64, ~8 ulp, on a template row's scale."""
    import torch

    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits
    from bbhx_b200.synthetic import data_grid, draw_params

    f = data_grid(tobs, lo, hi)
    if nudge:
        f[len(f) // 3] = np.nextafter(f[len(f) // 3], 1.0)
    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))
    P = draw_params(batch, tobs, 5 + length)
    P[11] = np.random.default_rng(length).uniform(0.6, 0.9, batch) * tobs * YEAR
    kw = dict(t_obs_start=0.0, t_obs_end=tobs, length=length, modes=modes)
    got, starts, lens = wave(*P, freqs=f, **kw)
    fd = torch.as_tensor(f, device="cuda")
    buf, c1, c2, c3, x, ts, te = wave._spline_set(tuple(P), 0.0, tobs, length, modes)
    B, M = batch, wave.num_modes
    x, y, c1, c2, c3 = (a.reshape(-1, B, M, length) for a in (x, buf, c1, c2, c3))
    eps = 8.0 * 2.0 ** -53 * 2.0 * np.pi * f[-1] * tobs * YEAR
    for b in range(B):
        st, n = int(starts[b]), int(lens[b])
        a, z = (int(torch.searchsorted(fd, v.reshape(1), right=True)) for v in (x[0, b].min(), x[0, b].max()))
        assert (st, n) == (a, z - a)
        if not n:
            continue
        ref = _interp_tdi(fd, x[0, b], y[:, b], (c1[:, b], c2[:, b], c3[:, b]), ts[b], te[b], st, n)
        for c in range(3):
            d = (got[b][c] - ref[c]).abs().max() / ref[c].abs().max()
            print(b, c, float(d), eps)
            assert d <= eps + 1e-12
