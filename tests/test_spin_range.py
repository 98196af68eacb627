"""Spins out of range: the row of the ringdown tables that the kernels read stays inside the tables
(the check of the spins is read after the launches on several paths), and
HeterodynedLikelihood.get_ll refuses such parameters before it launches or keeps anything."""
import math

import numpy as np
import pytest


def _row():
    from bbhx_b200 import _lib, build_ext

    build_ext.build()
    return _lib.lib().bbhx_selftest_qnm_row


def test_table_row_is_the_knot_interval_and_stays_in_the_table():
    row = _row()
    last, step = 1000, 0.002
    for fs in np.concatenate([np.linspace(-1.0, 1.0, 4001), np.nextafter(np.arange(-499, 500) * step, -2.0)]):
        fs = float(fs)
        assert row(fs, step, last) == int((fs - (-1.0)) / step)  # final spins of the model: unchanged
    for fs in (1.0000001, 1.066, 1.2, 5.0, 50.0, 1e9, 1e300, math.inf):
        assert row(fs, step, last) == last
    for fs in (-1.0000001, -1.2, -5.0, -50.0, -1e9, -1e300, -math.inf, math.nan):
        assert row(fs, step, last) == 0


class _Launched(Exception):
    pass


class _Template:
    def heterodyne_sums(self, *args, **kwargs):
        raise _Launched


def _likelihood():
    from bbhx_b200 import HeterodynedLikelihood

    het = HeterodynedLikelihood.__new__(HeterodynedLikelihood)
    het.precision = "fp64"
    het.template_gen, het.template_gen_kwargs = _Template(), {}
    het.freqs = het._h0_flat = het.data_constants = None
    het.hdyn_d_h, het.hdyn_h_h, het._last, het._h_sparse = "d_h", "h_h", "last", "sparse"
    return het


@pytest.mark.parametrize("row,value,message", [(2, 1.2, "chi1z"), (3, -1.0000001, "chi2z"), (2, np.inf, "chi1z")])
def test_heterodyned_refuses_spins_before_any_launch(row, value, message):
    het = _likelihood()
    P = np.full((12, 3), 0.5)
    P[row, 1] = value
    with pytest.raises(ValueError, match=message):
        het.get_ll(P)
    assert (het.hdyn_d_h, het.hdyn_h_h, het._last, het._h_sparse) == ("d_h", "h_h", "last", "sparse")


def test_nan_spins_pass_and_hide_nothing():
    from bbhx_b200.waveforms.phenomhm import raise_chi_range

    spins = np.array([[0.1, np.nan, -1.0], [1.0, np.nan, 0.3]])
    raise_chi_range(spins)
    raise_chi_range(spins[:, :0])
    spins[1, 2] = -1.5
    with pytest.raises(ValueError, match="chi2z"):
        raise_chi_range(spins)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("on_device,copies", [(False, 1), (True, 1), (False, 2100)])
def test_heterodyned_is_as_before_after_a_refused_call(golden, golden_data, precision, on_device,
                                                       copies):
    import torch

    from bbhx_b200 import AET1SensitivityMatrix, BBHWaveformFD, EqualArmlengthOrbits
    from bbhx_b200 import HeterodynedLikelihood, _lib

    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))
    kw = dict(t_obs_start=0.0, t_obs_end=golden_data["tobs"])
    het = HeterodynedLikelihood(wave, golden_data["f"], golden_data["data"], golden["params"][:, 0], 128,
                                template_gen_kwargs=dict(kw), reference_gen_kwargs=dict(kw, length=1024),
                                sens_mat=AET1SensitivityMatrix(golden_data["f"], tdi2=True),
                                precision=precision)
    P = np.tile(golden["het_walkers"], (1, copies))  # 8 walkers; 16800 are checked on the device
    as_given = (lambda a: torch.as_tensor(a, device="cuda")) if on_device else (lambda a: a)
    ref = het.get_ll(as_given(P), **kw).copy()
    d_h, last = het.hdyn_d_h.clone(), het._last
    take = _lib.lib().bbhx_take_status
    take(_lib.stream())
    bad = P.copy()
    bad[2, 0] = 1.2
    with pytest.raises(ValueError, match="chi1z"):
        het.get_ll(as_given(bad), **kw)
    assert take(_lib.stream()) == 0
    assert torch.equal(het.hdyn_d_h, d_h) and het._last is last
    np.testing.assert_array_equal(het.get_ll(as_given(P), **kw), ref)
