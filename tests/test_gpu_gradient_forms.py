"""The gradient's contraction (csrc/gradient_model.cuh, csrc/response_adjoint.cuh) at the sizes and
options where it branches: point counts around a warp's 32 and around the split of a (binary, mode)
over several warps, one mode and six, XYZ and AET, both TDI generations, and a source along an arm
(the series form of 1 / (1 - k.n)).  Oracle: central finite differences of the FP64 lnL with the
steps of tests/test_gpu_gradient.py (ten times them for the angles, whose phases move least, against
the rounding of lnL over the step) and twice those, without the h^2 term (the phase moves by 0.1 rad
per step in some spins: that term alone is 2e-4 there), and its bound (1e-4 relative plus
1e-7 of the largest scaled component)."""
import numpy as np
import pytest

from test_gpu_gradient import ROWS, _check, _steps

pytestmark = pytest.mark.gpu


def _extrapolated_fd(fn, P):
    """fn: [12, B] -> lnL [B]; returns [B, 11] central differences without their h^2 term."""
    B = P.shape[1]
    steps = np.array([_steps(P[:, b]) for b in range(B)])
    steps[:, 5:10] *= 10.0  # phi_ref, inc, lam, beta, psi
    out = np.zeros((B, len(ROWS)))
    for k, r in enumerate(ROWS):
        fd = []
        for h in (2.0 * steps[:, k], steps[:, k]):
            Pp, Pm = P.copy(), P.copy()
            Pp[r] += h
            Pm[r] -= h
            fd.append((fn(Pp) - fn(Pm)) / (2 * h))
        out[:, k] = (4.0 * fd[1] - fd[0]) / 3.0
    return out


def _wave(tdi, tdi2):
    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits

    return BBHWaveformFD(amp_phase_kwargs=dict(run_phenomd=False),
                         response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag=tdi, tdi2=tdi2))


def _injection(wave, center, golden_data, kw):
    return wave(*[np.atleast_1d(v) for v in center], freqs=golden_data["f"], length=1024, fill=True,
                direct=False, **kw)[0].cpu().numpy()


def _along_arm(center):
    from bbhx_b200 import EqualArmlengthOrbits

    n = EqualArmlengthOrbits().get_normal_unit_vec(np.array([center[11]]), 23)[0]
    n /= np.linalg.norm(n)
    center[8], center[9] = np.arctan2(-n[1], -n[0]) % (2 * np.pi), np.arcsin(-n[2])
    return center


@pytest.mark.parametrize("length,batch,modes,tdi,tdi2,arm", [
    (5, 1, [(2, 2)], "AET", True, False),
    (32, 3, [(2, 2), (2, 1)], "AET", False, False),
    (33, 2, None, "XYZ", False, False),
    (97, 2, None, "XYZ", True, False),
    (128, 2, None, "AET", True, True),
    (300, 500, [(2, 2), (3, 3), (4, 4)], "AET", True, False),
])
def test_heterodyned(golden, golden_data, length, batch, modes, tdi, tdi2, arm):
    from bbhx_b200 import AET1SensitivityMatrix, HeterodynedLikelihood
    from bbhx_b200.synthetic import perturb_params

    wave = _wave(tdi, tdi2)
    kw = dict(t_obs_start=0.0, t_obs_end=golden_data["tobs"])
    if modes is not None:
        kw["modes"] = modes
    center = golden["params"][:, 0].copy()
    if arm:
        center = _along_arm(center)
    data = _injection(wave, center, golden_data, kw) + golden_data["data"]
    het = HeterodynedLikelihood(wave, golden_data["f"], data, center, length,
                                template_gen_kwargs=dict(kw), reference_gen_kwargs=dict(kw, length=1024),
                                sens_mat=AET1SensitivityMatrix(golden_data["f"], tdi2=tdi2))
    P = perturb_params(center, batch, 7, rel_mass=1e-4, abs_spin_angle=1e-3, t_ref_s=1.0)
    grad = het.get_ll_and_grad(P, **kw)[1].cpu().numpy()
    _check(grad, _extrapolated_fd(lambda Q: het.get_ll(Q, **kw), P), P)


@pytest.mark.parametrize("length,batch,modes,tdi,tdi2,arm", [
    (33, 2, [(2, 2)], "AET", True, False),
    (100, 1, None, "XYZ", True, False),
    (257, 2, None, "XYZ", False, True),
    (512, 3, None, "AET", True, True),
])
def test_direct(golden, golden_data, length, batch, modes, tdi, tdi2, arm):
    from bbhx_b200 import Likelihood
    from bbhx_b200.synthetic import perturb_params

    wave = _wave(tdi, tdi2)
    kw = dict(t_obs_start=0.0, t_obs_end=golden_data["tobs"])
    if modes is not None:
        kw["modes"] = modes
    center = golden["params"][:, 0].copy()
    if arm:
        center = _along_arm(center)
    data = _injection(wave, center, golden_data, kw) + golden_data["data"]
    like = Likelihood(wave, golden_data["f"], data, golden_data["psd"])
    P = perturb_params(center, batch, 7, rel_mass=1e-4, abs_spin_angle=1e-3, t_ref_s=1.0)
    kw["length"] = length
    grad = like.get_ll_and_grad(P, **kw)[1].cpu().numpy()
    _check(grad, _extrapolated_fd(lambda Q: like.get_ll(Q, **kw), P), P)
