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
