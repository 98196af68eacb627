"""A source's <d|h> and <h|h> do not depend on the other sources of the call.  The number of
sources chooses the size of the fused kernels' work items (fused_tile, csrc/likelihood.cu: 256 bins
for one source, up to 4096 mixed and 8192 FP64 for hundreds), so a source is evaluated alone, in a
small and in a large batch, on grids whose low end holds more than 8 segments per 4096 bins (the
mixed form walks those) and whose upper bins lie in staged segments, at ragged band edges and
segment counts.

Tolerance: the mixed form evaluates every (bin, mode) with the same arithmetic whatever the item,
and only the FP64 sums over bins are taken in another order: 4 sum |d| |w h| over the bins is at
most sqrt(<d|d> <h|h>), a lane adds some hundred terms and the trees a few dozen, so the order moves
a sum by less than 1e3 * 2^-53 ~ 1e-13 of that; 1e-12 is asked for.  In 32 bits a change of the
arithmetic itself is 1e-8 and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

YEAR = 31558149.763545603


def _sums(like, P, kw):
    like.get_ll(P, **kw)
    return like.d_h.cpu().numpy().copy(), like.h_h.cpu().numpy().real.copy()


def _problem(tobs, lo, hi, batch, seed):
    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits, Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import data_grid, draw_params, gaussian_noise, notch_tdi_zeros

    f = data_grid(tobs, lo, hi)
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    data = gaussian_noise(psd, f[1] - f[0], seed)
    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))
    P = draw_params(batch, tobs, seed + 1)
    P[11] = np.random.default_rng(seed).uniform(0.75, 0.9, batch) * tobs * YEAR
    return Likelihood(wave, f, data, psd), P


@pytest.mark.parametrize("tobs,lo,hi,length,modes,batch", [
    (0.1, 1e-5, 0.1, 1024, None, 200),
    (0.1, 1e-5, 0.1, 256, [(2, 2), (3, 3), (2, 1)], 200),
    (0.31, 3.3e-5, 8.1e-2, 777, None, 90),
    (0.06, 1e-5, 0.03, 1500, [(2, 2)], 900),
])
def test_mixed_source_alone_equals_source_in_a_batch(tobs, lo, hi, length, modes, batch):
    like, P = _problem(tobs, lo, hi, batch, 31 + length)
    like.precision = "mixed"
    kw = dict(length=length, modes=modes, t_obs_start=0.0, t_obs_end=tobs)
    dh, hh = _sums(like, P, kw)
    for sel in ([0], [1], [2], [3], list(range(11))):
        d1, h1 = _sums(like, P[:, sel], kw)
        scale = np.sqrt(like.d_d * hh[sel])
        print(len(sel), np.max(np.abs(d1 - dh[sel]) / scale), np.max(np.abs(h1 - hh[sel]) / hh[sel]))
        assert np.all(np.abs(d1 - dh[sel]) <= 1e-12 * scale)
        assert np.all(np.abs(h1 - hh[sel]) <= 1e-12 * hh[sel])
