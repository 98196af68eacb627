"""TDI response of sources along a LISA arm, where 1 - (k.n)^2 of a link goes to zero and the
response changes from the addition theorem to the plain sinc form (csrc/response_model.cuh,
sinc_pair), against the numpy oracle.  Tolerance: 1e-10 of each transfer's scale, as in the
parity tests (rounding of ~1e-16 / (1 - k.n) on terms that themselves scale with 1 - (k.n)^2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tdi", ["AET", "XYZ"])
@pytest.mark.parametrize("link", [12, 23, 31])
@pytest.mark.parametrize("offset", [0.0, 3e-4, 9.5e-4, 1.05e-3, 1e-2])
def test_source_along_an_arm(tdi, link, offset):
    import torch

    from bbhx_b200 import EqualArmlengthOrbits, LISATDIResponse
    from oracle.kernels_np import FastLISAResponse

    orbits = EqualArmlengthOrbits()
    t0, L = 3.3e6, 200
    n = orbits.get_normal_unit_vec(np.array([t0]), link)[0]
    lam, beta = np.arctan2(-n[1], -n[0]), np.arcsin(-n[2] / np.linalg.norm(n)) + offset
    freqs = np.geomspace(1e-5, 0.1, L)
    modes = [(2, 2), (3, 3)]
    inc, psi, phi = 0.7, 0.3, 1.1
    resp = LISATDIResponse(TDItag=tdi, orbits=orbits, tdi2=True)
    phase = torch.zeros((1, 2, L), dtype=torch.float64, device="cuda")
    tf = torch.full((1, 2, L), t0, dtype=torch.float64, device="cuda")
    f = np.tile(freqs, (1, 2, 1))
    resp(f, np.array([inc]), np.array([lam]), np.array([beta]), np.array([psi]), np.array([phi]), L,
         modes=modes, phase=phase, tf=tf)
    got = [getattr(resp, "transferL%d" % c)[0].cpu().numpy() for c in (1, 2, 3)]
    ref = FastLISAResponse()
    ref.add_orbit_information(*orbits.pycppdetector_args)
    for i, (ell, mm) in enumerate(modes):
        k, H = ref.mode_matrix(ell, mm, phi, inc, lam, beta, psi)
        T = ref.transfer(H, k, freqs, np.full(L, t0), 1 if tdi == "XYZ" else 2, False, True)
        for c in range(3):
            scale = np.max(np.abs(T[c]))
            d = np.max(np.abs(got[c][i] - T[c])) / scale
            print(tdi, link, offset, (ell, mm), c, d)
            assert d <= 1e-10
