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
