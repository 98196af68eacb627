"""The spline solve (csrc/tridiag.cuh) at the lengths and quantity counts where its levels change
hands, and the support search (csrc/likelihood.cu, warp_count_le) around its 32 probes per round.

Oracles: scipy's not-a-knot cubic spline, with 1e-11 of max |y| at the segment middles (the rows are
diagonally dominant by 2, so the slopes carry a few rounding errors of the divided differences, and
h * slope is at most of the order of y here), and numpy.searchsorted, exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quantities", [1, 9, 12])
@pytest.mark.parametrize("length", [4, 5, 15, 16, 17, 64, 65, 66, 127, 129, 513, 1000, 1025, 1791, 2600])
def test_spline_solve(length, quantities):
    import torch
    from scipy.interpolate import CubicSpline

    from bbhx_b200 import _lib

    rng = np.random.default_rng(length * 17 + quantities)
    systems = 3
    x = np.geomspace(1e-4, 1e-1, length) * (1 + 0.1 * rng.random((systems, 1)))
    y = np.stack([np.cos((p + 1) * np.log(x / 1e-4)) + p for p in range(quantities)])
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda").contiguous()
    xd, yd = dev(x), dev(y)
    out = [torch.empty_like(yd) for _ in range(4)]
    _lib.call("bbhx_interpolate", _lib.dptr(xd), _lib.dptr(yd), *[_lib.dptr(o) for o in out], length,
              quantities, 1, systems, _lib.stream())
    c1, c2, c3 = [o.cpu().numpy() for o in out[1:]]
    mid = 0.5 * (x[:, 1:] - x[:, :-1])
    for p in range(quantities):
        for s in range(systems):
            h = mid[s]
            got = y[p, s, :-1] + h * (c1[p, s, :-1] + h * (c2[p, s, :-1] + h * c3[p, s, :-1]))
            ref = CubicSpline(x[s], y[p, s])(x[s, :-1] + h)
            assert np.max(np.abs(got - ref)) <= 1e-11 * np.max(np.abs(y[p, s]))


@pytest.mark.parametrize("bins", [1, 2, 31, 32, 33, 1023, 1024, 1025, 1057, 40000])
@pytest.mark.parametrize("uniform", [True, False])
def test_support(bins, uniform):
    import torch

    from bbhx_b200 import _lib

    rng = np.random.default_rng(bins)
    f = np.arange(1, bins + 1) * 1e-5 if uniform else np.sort(rng.random(bins) * bins * 1e-5)
    B, M, L = 64, 2, 8
    edge = rng.choice(f, (B, 2))
    lo = np.where(rng.random(B) < 0.3, edge[:, 0], rng.uniform(0.5 * f[0], 1.2 * f[-1], B))
    hi = np.maximum(lo, np.where(rng.random(B) < 0.3, edge[:, 1], lo * rng.uniform(1, 5, B)))
    x = np.sort(np.concatenate([lo[:, None], hi[:, None], lo[:, None] + (hi - lo)[:, None] *
                                rng.random((B, M * L - 2))], axis=1), axis=1).reshape(B, M, L)
    xd = torch.tensor(x, dtype=torch.float64, device="cuda")
    fd = torch.tensor(f, dtype=torch.float64, device="cuda")
    start = torch.empty(B, dtype=torch.int32, device="cuda")
    length = torch.empty_like(start)
    _lib.call("bbhx_template_support", _lib.dptr(start), _lib.dptr(length), _lib.dptr(xd), M, L, B,
              _lib.dptr(fd), bins, _lib.stream())
    a = np.searchsorted(f, x.min(axis=(1, 2)), side="right")
    b = np.searchsorted(f, x.max(axis=(1, 2)), side="right")
    np.testing.assert_array_equal(start.cpu().numpy(), a)
    np.testing.assert_array_equal(length.cpu().numpy(), b - a)
