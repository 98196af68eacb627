"""A binary whose whole knot range falls between two data bins has no bins: its sums are exactly zero,
whatever its neighbours in the call are, on uniform and other grids, FP64 and mixed.  (The item of the
tile that holds its place must be skipped: its segment table entries are placeholders, so the walk of
the panels would start on segments that nobody copied.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("bins,place", [(1000, 500), (256, 0), (256, 254), (513, 255), (700, 511)])
def test_knots_between_two_bins(bins, place, uniform, mixed):
    import torch

    from bbhx_b200 import _lib

    rng = np.random.default_rng(bins + place)
    f = np.arange(100, 100 + bins) * 1e-5
    if not uniform:
        f[bins // 2] = np.nextafter(f[bins // 2], 1.0)
    B, M, L = 3, 2, 8
    x = np.empty((B, M, L))
    x[0::2] = np.linspace(0.7 * f[0], 1.1 * f[-1], L)
    x[1] = np.linspace(f[place] + 2e-6, f[place] + 8e-6, L)
    y = rng.standard_normal((9, B, M, L))
    y[2] = 5.0  # t(f), inside the observation [0, 10]
    c = 1e-3 * rng.standard_normal((3, 9, B, M, L))
    c[:, 2] = 0.0
    dev = lambda a: torch.tensor(a, device="cuda").contiguous()
    fd, xd, yd, c1, c2, c3 = dev(f), dev(x), dev(y), *map(dev, c)
    data = dev(rng.standard_normal((3, bins)) + 1j * rng.standard_normal((3, bins)))
    noise = dev(rng.random((3, bins)) + 0.5)
    d32, n32 = data.to(torch.complex64), noise.to(torch.float32)
    ts, te = dev(np.zeros(B)), dev(np.full(B, 10.0))
    d_h = torch.full((B,), 7.0, dtype=torch.complex128, device="cuda")
    h_h = d_h.clone()
    p, z = _lib.dptr, _lib._VP(0)
    _lib.call("bbhx_direct_like_fused", p(d_h), p(h_h), p(fd), p(data), p(noise), bins, p(xd), p(yd),
              p(c1), p(c2), p(c3), p(ts), p(te), M, L, B, int(mixed), p(d32) if mixed else z,
              p(n32) if mixed else z, _lib.stream())
    d_h, h_h = d_h.cpu().numpy(), h_h.cpu().numpy()
    assert d_h[1] == 0.0 and h_h[1] == 0.0
    assert np.all(np.isfinite(d_h)) and np.all(h_h[[0, 2]].real > 0.0)
