"""The spline solve where the block's size and the sharing of right-hand sides change: block sizes of
32 to 384 threads by length, number of systems and shared memory (csrc/spline.cu, spline_threads), and
teams of one to twelve warps to a right-hand side (csrc/tridiag.cuh).  Oracle and tolerance as in
test_gpu_spline_edges.py: scipy's not-a-knot spline at the segment middles, 1e-11 of max |y|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("systems", [2, 400])
@pytest.mark.parametrize("quantities", [1, 2, 3, 4, 5, 7, 9])
@pytest.mark.parametrize("length", [4, 33, 64, 65, 130, 320, 321, 700, 701, 1024, 1300, 3000])
def test_spline_solve(length, quantities, systems):
    import torch
    from scipy.interpolate import CubicSpline

    from bbhx_b200 import _lib

    rng = np.random.default_rng(length * 31 + quantities)
    x = np.geomspace(1e-4, 1e-1, length) * (1 + 0.1 * rng.random((systems, 1)))
    y = np.stack([np.cos((p + 1) * np.log(x / 1e-4)) + p for p in range(quantities)])
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda").contiguous()
    xd, yd = dev(x), dev(y)
    out = [torch.full_like(yd, np.nan) for _ in range(4)]
    _lib.call("bbhx_interpolate", _lib.dptr(xd), _lib.dptr(yd), *[_lib.dptr(o) for o in out], length,
              quantities, 1, systems, _lib.stream())
    c1, c2, c3 = [o.cpu().numpy() for o in out[1:]]
    assert np.all(np.isfinite(c1)) and np.all(np.isfinite(c2[:, :, :-1])) and np.all(np.isfinite(c3[:, :, :-1]))
    for s in {0, 1, systems // 2, systems - 1}:
        h = 0.5 * (x[s, 1:] - x[s, :-1])
        for p in range(quantities):
            got = y[p, s, :-1] + h * (c1[p, s, :-1] + h * (c2[p, s, :-1] + h * c3[p, s, :-1]))
            ref = CubicSpline(x[s], y[p, s])(x[s, :-1] + h)
            assert np.max(np.abs(got - ref)) <= 1e-11 * np.max(np.abs(y[p, s]))
