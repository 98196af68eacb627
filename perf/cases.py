"""What this package is measured on: likelihoods, gradients and templates of massive-black-hole
binaries through the package's public classes, over the sizes a LISA analysis uses.

Kinds of case (``case["kind"]``):

* ``lnl``       ``Likelihood.get_ll``: the direct likelihood on the whole data stream;
* ``lnl_grad``  ``Likelihood.get_ll_and_grad``: the same with its eleven derivatives;
* ``het``       ``HeterodynedLikelihood.get_ll``: relative binning, many walkers near a reference;
* ``het_grad``  ``HeterodynedLikelihood.get_ll_and_grad``;
* ``fill``      ``BBHWaveformFD`` with ``fill=True, combine=True``: an injected data stream;
* ``sparse``    ``BBHWaveformFD`` with ``direct=True``: templates on a short frequency grid.

``exact`` restates the whole path (PhenomHM, TDI response, splines, inner products) in plain
64-bit torch, with autograd for the derivatives.
"""
import math

import numpy as np
import torch

YEAR = 31558149.763545603
F_LO, F_HI = 1e-5, 0.1
ALL_MODES = [(2, 2), (3, 3), (4, 4), (2, 1), (3, 2), (4, 3)]
GRAD_ROWS = [0, 1, 2, 3, 4, 5, 7, 8, 9, 10, 11]


def listed():
    return [
        # one source in a month of data, the dominant mode: the smallest call a user makes
        dict(name="lnl_one_small", kind="lnl", batch=1, tobs=0.1, length=256, modes="22",
             precision="fp64"),
        # one source in a year of data: a step of a serial sampler
        dict(name="lnl_one_year", kind="lnl", batch=1, tobs=1.0, length=1024, modes="all",
             precision="fp64"),
        # the walkers of an ensemble sampler, odd sizes, three modes
        dict(name="lnl_walkers", kind="lnl", batch=53, tobs=0.31, length=777, modes="22,33,44",
             precision="fp64"),
        # the benchmark's batch: all walkers of a parallel-tempered sampler in a year of data
        dict(name="lnl_batch_year", kind="lnl", batch=1024, tobs=1.0, length=1024, modes="all",
             precision="fp64"),
        # the mixed-precision option on an ordinary batch
        dict(name="lnl_mixed", kind="lnl", batch=150, tobs=0.5, length=1024, modes="all",
             precision="mixed"),
        # derivatives of the direct likelihood for a set of Hamiltonian chains
        dict(name="lnl_grad", kind="lnl_grad", batch=128, tobs=0.25, length=512, modes="all"),
        # a few walkers of a heterodyned run
        dict(name="het_few", kind="het", batch=24, tobs=0.25, length=128, precision="fp64"),
        # a large ensemble of heterodyned walkers
        dict(name="het_batch", kind="het", batch=16384, tobs=0.25, length=128, precision="fp64"),
        # the mixed-precision option, a finer and odd grid
        dict(name="het_mixed", kind="het", batch=4099, tobs=0.25, length=193, precision="mixed"),
        # derivatives of the heterodyned likelihood
        dict(name="het_grad", kind="het_grad", batch=2048, tobs=0.25, length=128),
        # an injection of several sources into a year of data
        dict(name="fill_year", kind="fill", batch=5, tobs=1.0, length=1024, modes="all", tdi="AET"),
        # templates on a frequency grid of the user's, as for plots, fits and signal-to-noise maps
        dict(name="sparse_templates", kind="sparse", batch=300, tobs=1.0, length=1000,
             modes="all", tdi="AET"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _count(rng, lo, hi):
    return min(hi, max(lo, int(round(_log(rng, lo, hi)))))


def draw(rng):
    kind = rng.choice(["lnl", "lnl", "lnl", "lnl_grad", "het", "het", "het_grad", "fill", "sparse"])
    modes = rng.choice(["all", "all", "all", "22", "22,33,44", "22,21,33"])
    if kind in ("lnl", "lnl_grad"):
        grad = kind == "lnl_grad"
        tobs = round(_log(rng, 0.05, 0.4 if grad else 1.0), 4)
        case = dict(kind=kind, batch=_count(rng, 1, 200 if grad else 900), tobs=tobs,
                    length=_count(rng, 250, 1500), modes=modes)
        return case if grad else dict(case, precision=rng.choice(["fp64", "fp64", "fp64", "mixed"]))
    if kind in ("het", "het_grad"):
        grad = kind == "het_grad"
        case = dict(kind=kind, batch=_count(rng, 1, 4000 if grad else 20000),
                    tobs=round(_log(rng, 0.1, 0.3), 4), length=_count(rng, 60, 320))
        return case if grad else dict(case, precision=rng.choice(["fp64", "fp64", "mixed"]))
    tdi = rng.choice(["AET", "AET", "XYZ"])
    if kind == "fill":
        return dict(kind=kind, batch=_count(rng, 1, 12), tobs=round(_log(rng, 0.1, 1.0), 4),
                    length=_count(rng, 500, 1500), modes=modes, tdi=tdi)
    return dict(kind=kind, batch=_count(rng, 1, 600), tobs=1.0, length=_count(rng, 100, 3000),
                modes=modes, tdi=tdi)


# ------------------------------------------------------------------------------- inputs
def _mode_list(case):
    """None (all modes) or the mode list a user passes."""
    names = case.get("modes", "all")
    return None if names == "all" else [(int(n[0]), int(n[1])) for n in names.split(",")]


def _draw_sources(case, n, rng):
    """[12, n] parameters from the priors of massive-black-hole binaries; the merger lies in the
    last quarter of the observation, far enough from its end that the light travel time over
    the orbit does not move it out."""
    total, q = 10.0 ** rng.uniform(5.0, 7.0, n), rng.uniform(0.1, 1.0, n)
    gpc = 1e9 * 3.0856775814913674e16
    return np.array([
        total / (1.0 + q), total * q / (1.0 + q), rng.uniform(-0.9, 0.9, n),
        rng.uniform(-0.9, 0.9, n), rng.uniform(10.0, 100.0, n) * gpc,
        rng.uniform(0.0, 2.0 * np.pi, n), np.zeros(n), np.arccos(rng.uniform(-1.0, 1.0, n)),
        rng.uniform(0.0, 2.0 * np.pi, n), np.arcsin(rng.uniform(-1.0, 1.0, n)),
        rng.uniform(0.0, np.pi, n), rng.uniform(0.75, 0.93, n) * case["tobs"] * YEAR])


def _walkers(center, n, rng):
    """[12, n] walkers around ``center``: the spread of a chain that has found its source."""
    out = np.repeat(center[:, None], n, axis=1)
    total = (center[0] + center[1]) * (1.0 + 1e-3 * rng.standard_normal(n))
    q = np.clip(center[1] / center[0] * (1.0 + 1e-3 * rng.standard_normal(n)), 0.05, 1.0)
    out[0], out[1] = total / (1.0 + q), total * q / (1.0 + q)
    for k in (2, 3, 5, 7, 8, 9, 10):
        out[k] += 1e-2 * rng.standard_normal(n)
    out[9] = np.clip(out[9], -0.5 * np.pi, 0.5 * np.pi)
    out[11] += 10.0 * rng.standard_normal(n)
    return out


def _inputs(case, seed):
    """Everything drawn from the seed: data grid, PSD, noise and parameters."""
    rng = np.random.default_rng(seed)
    df = 1.0 / (case["tobs"] * YEAR)
    out = {}
    if case["kind"] != "sparse":
        out["f"] = np.arange(math.ceil(F_LO / df), math.floor(F_HI / df) + 1) * df
    if case["kind"] in ("lnl", "lnl_grad", "het", "het_grad"):
        out["injection"] = _draw_sources(case, 1, rng)
        out["psd"] = _psd(out["f"])
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        noise = torch.randn((3, len(out["f"]), 2), generator=gen, dtype=torch.float64, device="cuda")
        psd = torch.as_tensor(out["psd"], device="cuda")
        sigma = torch.sqrt(torch.where(torch.isfinite(psd), psd, 0.0) / (4.0 * df))
        out["noise"] = sigma * torch.view_as_complex(noise)
    if case["kind"] in ("het", "het_grad"):
        out["params"] = _walkers(out["injection"][:, 0], case["batch"], rng)
    else:
        out["params"] = _draw_sources(case, case["batch"], rng)
    return out


def _psd(f):
    """A / E / T noise, second-generation TDI, the bins around its zeros left out."""
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import notch_tdi_zeros

    return notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))


def _kwargs(case):
    return dict(t_obs_start=0.0, t_obs_end=case["tobs"])


def prepare(case, seed):
    from bbhx_b200 import (AET1SensitivityMatrix, BBHWaveformFD, EqualArmlengthOrbits,
                           HeterodynedLikelihood, Likelihood)

    kind, x = case["kind"], _inputs(case, seed)
    wave = BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(),
                                              TDItag=case.get("tdi", "AET"), tdi2=True))
    kw = _kwargs(case)
    state = dict(kind=kind, params=x["params"], kw=dict(kw, modes=_mode_list(case)))
    if kind == "fill":
        state.update(wave=wave, freqs=torch.as_tensor(x["f"], device="cuda"))
        state["kw"]["length"] = case["length"]
        return state
    if kind == "sparse":
        state.update(wave=wave, freqs=torch.as_tensor(_sparse_grid(case), device="cuda"))
        return state
    data = x["noise"] + wave(*x["injection"], freqs=torch.as_tensor(x["f"], device="cuda"),
                             length=1024, fill=True, combine=True, **kw)
    if kind in ("lnl", "lnl_grad"):
        like = Likelihood(wave, x["f"], data, x["psd"], precision=case.get("precision", "fp64"))
        state["kw"]["length"] = case["length"]
    else:
        like = HeterodynedLikelihood(
            wave, x["f"], data, x["injection"][:, 0], case["length"], template_gen_kwargs=dict(kw),
            reference_gen_kwargs=dict(kw, length=1024), precision=case.get("precision", "fp64"),
            sens_mat=AET1SensitivityMatrix(x["f"], tdi2=True, notch=True))
        state["kw"] = kw
    state["like"] = like
    if kind in ("lnl_grad", "het_grad"):  # gradient-based samplers keep their state on the GPU
        state["params"] = torch.as_tensor(x["params"], device="cuda")
    return state


def _sparse_grid(case):
    return np.logspace(-4.0, -1.3, case["length"])


def run(state):
    kind, kw = state["kind"], state["kw"]
    if kind == "lnl":
        like = state["like"]
        return {"lnl": like.get_ll(state["params"], **kw), "d_h": like.d_h, "h_h": like.h_h}
    if kind == "het":
        like = state["like"]
        return {"lnl": like.get_ll(state["params"], **kw), "d_h": like.hdyn_d_h,
                "h_h": like.hdyn_h_h}
    if kind in ("lnl_grad", "het_grad"):
        lnl, grad = state["like"].get_ll_and_grad(state["params"], **kw)
        return {"lnl": lnl, "grad": grad}
    if kind == "fill":
        return state["wave"](*state["params"], freqs=state["freqs"], fill=True, combine=True, **kw)
    return state["wave"](*state["params"], freqs=state["freqs"], direct=True, compress=True, **kw)


def work(case):
    """Inputs and outputs once; a waveform model and response of about 600 operations per sparse
    point; and 36 operations (three complex products with the data, three squares) per binary
    and data bin, about ten times that with derivatives."""
    b, points = case["batch"], case["length"] * len(_mode_list(case) or ALL_MODES)
    n = int((F_HI - F_LO) * case["tobs"] * YEAR)
    kind, model = case["kind"], 600.0 * b * points
    params = 96.0 * b
    if kind == "lnl":
        return {"bytes": 80.0 * n + params + 40.0 * b, "flops": model + 36.0 * b * n}
    if kind == "lnl_grad":
        return {"bytes": 80.0 * n + params + 96.0 * b, "flops": 12.0 * model + 100.0 * b * n}
    if kind in ("het", "het_grad"):
        grad = kind == "het_grad"
        return {"bytes": 250.0 * case["length"] + params + (96.0 if grad else 40.0) * b,
                "flops": (12.0 if grad else 1.0) * model}
    if kind == "fill":
        return {"bytes": 56.0 * n + params, "flops": model + 60.0 * b * n}
    return {"bytes": 48.0 * b * case["length"] + params, "flops": model}


# ------------------------------------------------------- the same path in plain 64-bit torch
# PhenomD fits (Khan et al. 2016, table V): coefficients of 1, eta, then xi, xi eta, xi eta^2, and
# the same for xi^2 and xi^3, with xi = chi - 1.
_FITS = {
    "rho1": (3931.8979897196696, -17395.758706812805, 3132.375545898835, 343965.86092361377,
             -1.2162565819981997e6, -70698.00600428853, 1.383907177859705e6,
             -3.9662761890979446e6, -60017.52423652596, 803515.1181825735, -2.091710365941658e6),
    "rho2": (-40105.47653771657, 112253.0169706701, 23561.696065836168, -3.476180699403351e6,
             1.137593670849482e7, 754313.1127166454, -1.308476044625268e7,
             3.6444584853928134e7, 596226.612472288, -7.4277901143564405e6,
             1.8928977514040343e7),
    "rho3": (83208.35471266537, -191237.7264145924, -210916.2454782992, 8.71797508352568e6,
             -2.6914942420669552e7, -1.9889806527362722e6, 3.0888029960154563e7,
             -8.390870279256162e7, -1.4535031953446497e6, 1.7063528990822166e7,
             -4.2748659731120914e7),
    "gamma1": (0.006927402739328343, 0.03020474290328911, 0.006308024337706171,
               -0.12074130661131138, 0.26271598905781324, 0.0034151773647198794,
               -0.10779338611188374, 0.27098966966891747, 0.0007374185938559283,
               -0.02749621038376281, 0.0733150789135702),
    "gamma2": (1.010344404799477, 0.0008993122007234548, 0.283949116804459, -4.049752962958005,
               13.207828172665366, 0.10396278486805426, -7.025059158961947, 24.784892370130475,
               0.03093202475605892, -2.6924023896851663, 9.609374464684983),
    "gamma3": (1.3081615607036106, -0.005537729694807678, -0.06782917938621007,
               -0.6689834970767117, 3.403147966134083, -0.05296577374411866,
               -0.9923793203111362, 4.820681208409587, -0.006134139870393713,
               -0.38429253308696365, 1.7561754421985984),
    "v2": (0.8149838730507785, 2.5747553517454658, 1.1610198035496786, -2.3627771785551537,
           6.771038707057573, 0.7570782938606834, -2.7256896890432474, 7.1140380397149965,
           0.1766934149293479, -0.7978690983168183, 2.1162391502005153),
    "sigma1": (2096.551999295543, 1463.7493168261553, 1312.5493286098522, 18307.330017082117,
               -43534.1440746107, -833.2889543511114, 32047.31997183187, -108609.45037520859,
               452.25136398112204, 8353.439546391714, -44531.3250037322),
    "sigma2": (-10114.056472621156, -44631.01109458185, -6541.308761668722,
               -266959.23419307504, 686328.3229317984, 3405.6372187679685,
               -437507.7208209015, 1.6318171307344697e6, -7462.648563007646,
               -114585.25177153319, 674402.4689098676),
    "sigma3": (22933.658273436497, 230960.00814979506, 14961.083974183695,
               1.1940181342318142e6, -3.1042239693052764e6, -3038.166617199259,
               1.8720322849093592e6, -7.309145012085539e6, 42738.22871475411,
               467502.018616601, -3.064853498512499e6),
    "sigma4": (-14621.71522218357, -377812.8579387104, -9608.682631509726,
               -1.7108925257214056e6, 4.332924601416521e6, -22366.683262266528,
               -2.5019716386377467e6, 1.0274495902259542e7, -85360.30079034246,
               -570025.3441737515, 4.396844346849777e6),
    "beta1": (97.89747327985583, -42.659730877489224, 153.48421037904913, -1417.0620760768954,
              2752.8614143665027, 138.7406469558649, -1433.6585075135881, 2857.7418952430758,
              41.025109467376126, -423.680737974639, 850.3594335657173),
    "beta2": (-3.282701958759534, -9.051384468245866, -12.415449742258042, 55.4716447709787,
              -106.05109938966335, -11.953044553690658, 76.80704618365418, -155.33172948098394,
              -3.4129261592393263, 25.572377569952536, -54.408036707740465),
    "beta3": (-0.000025156429818799565, 0.000019750256942201327, -0.000018370671469295915,
              0.000021886317041311973, 0.00008250240316860033, 7.157371250566708e-6,
              -0.000055780000112270685, 0.00019142082884072178, 5.447166261464217e-6,
              -0.00003220610095021982, 0.00007974016714984341),
    "alpha1": (43.31514709695348, 638.6332679188081, -32.85768747216059, 2415.8938269370315,
               -5766.875169379177, -61.85459307173841, 2953.967762459948, -8986.29057591497,
               -21.571435779762044, 981.2158224673428, -3239.5664895930286),
    "alpha2": (-0.07020209449091723, -0.16269798450687084, -0.1872514685185499,
               1.138313650449945, -2.8334196304430046, -0.17137955686840617,
               1.7197549338119527, -4.539717148261272, -0.049983437357548705,
               0.6062072055948309, -1.682769616644546),
    "alpha3": (9.5988072383479, -397.05438595557433, 16.202126189517813, -1574.8286986717037,
               3600.3410843831093, 27.092429659075467, -1786.482357315139, 5152.919378666511,
               11.175710130033895, -577.7999423177481, 1808.730762932043),
    "alpha4": (-0.02989487384493607, 1.4022106448583738, -0.07356049468633846,
               0.8337006542278661, 0.2240008282397391, -0.055202870001177226,
               0.5667186343606578, 0.7186931973380503, -0.015507437354325743,
               0.15750322779277187, 0.21076815715176228),
    "alpha5": (0.9974408278363099, -0.007884449714907203, -0.059046901195591035,
               1.3958712396764088, -4.516631601676276, -0.05585343136869692,
               1.7516580039343603, -5.990208965347804, -0.017945336522161195,
               0.5965097794825992, -2.0608879367971804),
}
# Remnant quasi-normal modes (London & Fauchon-Jones 2019): offset, power of kappa in front,
# amplitudes and phases of the powers of kappa.
_QNM = {
    (2, 2): (1, 1.0, (1.557847, 1.95097051, 2.09971716, 1.41094660, 0.41063923),
             (2.903124, 5.920970, 2.760585, 5.914340, 2.795235)),
    (3, 3): (1, 1.5, (2.095657, 2.46964352, 2.66552551, 1.75836443, 0.49905688),
             (2.964973, 5.996734, 2.817591, 5.932693, 2.781658)),
    (4, 4): (1, 2.0, (2.658908, 2.97825567, 3.21842350, 2.12764967, 0.60338186),
             (3.002787, 6.050955, 2.877514, 5.989669, 2.830031)),
    (2, 1): (0, 0.0, (0.589113, 0.18896353, 1.15012965, 6.04585476, 11.12627777, 9.34711461,
                      3.03838318),
             (0.043525, 2.289868, 5.810057, 2.741967, 5.844130, 2.669372, 5.791518)),
    (3, 2): (0, 0.0, (1.022464, 0.24731213, 1.70468239, 0.94604882, 1.53189884, 2.28052668,
                      0.92150314),
             (0.004870, 0.665292, 3.138283, 0.163247, 5.703573, 2.685231, 5.841704)),
    (4, 3): (1, 1.5, (0.205046, 3.10333396, 4.23612166, 3.02890198, 0.90843949),
             (0.595328, 3.016200, 6.038842, 2.826239, 5.915164)),
}
_SHIFT = {1: 0.5 * math.pi, 2: 0.0, 3: -0.5 * math.pi, 4: math.pi}
_MTSUN, _MRSUN, _C, _AU, _ARM = (4.925491025873693e-06, 1476.6250615036158, 299792458.0,
                                 149597870700.0, 2.5e9)
_OMEGA_ORBIT, _OMEGA_FRAME = 1.9909865927683788e-07, 1.99098659277e-7
_EULER = 0.577215664901532860606512090082402431
_AMP_JOIN, _PHI_JOIN = 0.014, 0.018


def _tensor(v):
    return torch.as_tensor(np.asarray(v, dtype=np.float64), device="cuda")


def _cubic(x, y):
    """Not-a-knot cubic splines through y [Q, S, L] over x [S, L]: coefficients c0..c3."""
    h = x[:, 1:] - x[:, :-1]
    m = (y[..., 1:] - y[..., :-1]) / h
    a, b = h[:, :-1], h[:, 1:]
    d0, dl = x[:, 2] - x[:, 0], x[:, -1] - x[:, -3]
    diag = torch.cat([h[:, 1:2], 2.0 * (a + b), h[:, -2:-1]], dim=1)
    up = torch.cat([d0[:, None], a], dim=1)
    low = torch.cat([b, dl[:, None]], dim=1)
    A = torch.diag_embed(diag) + torch.diag_embed(up, 1) + torch.diag_embed(low, -1)
    first = ((h[:, 0] + 2 * d0) * h[:, 1] * m[..., 0] + h[:, 0] ** 2 * m[..., 1]) / d0
    last = (h[:, -1] ** 2 * m[..., -2] + (2 * dl + h[:, -1]) * h[:, -2] * m[..., -1]) / dl
    r = torch.cat([first[..., None], 3.0 * (b * m[..., :-1] + a * m[..., 1:]), last[..., None]],
                  dim=-1)
    s = torch.linalg.solve(A, r.permute(1, 2, 0)).permute(2, 0, 1)
    t = (s[..., :-1] + s[..., 1:] - 2.0 * m) / h
    return y[..., :-1], s[..., :-1], (m - s[..., :-1]) / h - t, t / h


class _PhenomD:
    """PhenomD amplitude and phase; coefficients carry a last axis of one for the frequencies."""

    def __init__(self, m1, m2, x1, x2, rd, dm, rho, tau):
        total = m1 + m2
        eta = m1 * m2 / total ** 2
        seta = torch.sqrt(1.0 - 4.0 * eta)
        chi = 0.5 * (x1 + x2) * (1.0 - 76.0 * eta / 113.0) + seta * 0.5 * (x1 - x2)
        self.eta, self.rd, self.dm, self.rho, self.tau = eta, rd, dm, rho, tau
        xi = chi - 1.0
        fit = {}
        for k, c in _FITS.items():
            poly = [c[2 + 3 * j] + c[3 + 3 * j] * eta + c[4 + 3 * j] * eta ** 2 for j in range(3)]
            fit[k] = c[0] + c[1] * eta + xi * (poly[0] + xi * (poly[1] + xi * poly[2]))
        pi, e2, e3 = math.pi, eta ** 2, eta ** 3
        a1, a2 = x1 ** 2, x2 ** 2
        self.amp0 = math.sqrt(2.0 / 3.0) * torch.sqrt(eta) / pi ** (1.0 / 6.0)
        self.ains = [
            (-969 + 1804 * eta) * pi ** (2.0 / 3.0) / 672.0,
            (x1 * (81 * (1 + seta) - 44 * eta) + x2 * (81 - 81 * seta - 44 * eta)) * pi / 48.0,
            (-27312085.0 - 10287648 * a2 - 10287648 * a1 * (1 + seta) + 10287648 * a2 * seta
             + 24 * (-1975055 + 857304 * a1 - 994896 * x1 * x2 + 857304 * a2) * eta
             + 35371056 * e2) * pi ** (4.0 / 3.0) / 8.128512e6,
            pi ** (5.0 / 3.0)
            * (x2 * (-285197 * (-1 + seta) + 4 * (-91902 + 1579 * seta) * eta - 35632 * e2)
               + x1 * (285197 * (1 + seta) - 4 * (91902 + 1579 * seta) * eta - 35632 * e2)
               + 42840 * (-1.0 + 4 * eta) * pi) / 32256.0,
            -(pi ** 2 * (-336 * (-3248849057.0 + 2943675504 * a1 - 3339284256 * x1 * x2
                                 + 2943675504 * a2) * e2
                         - 324322727232 * e3
                         - 7 * (-177520268561 + 107414046432 * a2 + 107414046432 * a1 * (1 + seta)
                                - 107414046432 * a2 * seta
                                + 11087290368 * (x1 + x2 + x1 * seta - x2 * seta) * pi)
                         + 12 * eta * (-545384828789 - 176491177632 * x1 * x2 + 202603761360 * a2
                                       + 77616 * a1 * (2610335 + 995766 * seta)
                                       - 77287373856 * a2 * seta + 5841690624 * (x1 + x2) * pi
                                       + 21384760320 * pi ** 2))) / 6.0085960704e10,
            fit["rho1"], fit["rho2"], fit["rho3"]]
        self.g1, self.g2, self.g3 = fit["gamma1"], fit["gamma2"], fit["gamma3"]
        below = self.g2 <= 1.0
        root = torch.where(below, torch.sqrt(torch.where(below, 1.0 - self.g2 ** 2, 1.0)), 0.0)
        self.peak = torch.abs(rd + dm * (-1.0 + root) * self.g3 / self.g2)
        # quartic of the intermediate amplitude in x = (f - f1) / (peak - f1)
        f1, width = _AMP_JOIN, self.peak - _AMP_JOIN
        powers = [2 / 3, 1.0, 4 / 3, 5 / 3, 2.0, 7 / 3, 8 / 3, 3.0]
        v1 = 1.0 + sum(c * f1 ** p for c, p in zip(self.ains, powers))
        d1 = sum(p * c * f1 ** (p - 1.0) for c, p in zip(self.ains, powers))
        v3 = self._amp_mrd(self.peak)
        s, off = self.dm * self.g3, self.peak - self.rd
        d3 = v3 * (-self.g2 / s - 2.0 * off / (off * off + s * s))
        k = torch.linalg.inv(_tensor([[1, 0, 0, 0, 0], [0, 1, 0, 0, 0],
                                      [1, 0.5, 0.25, 0.125, 0.0625], [1, 1, 1, 1, 1],
                                      [0, 1, 2, 3, 4]]))
        cond = [v1, d1 * width, fit["v2"], v3, d3 * width]
        self.mid = [sum(k[i, j] * cond[j] for j in range(5)) for i in range(5)]
        self.width = width
        self._phase_setup(m1 / total, m2 / total, x1, x2, fit)

    def _phase_setup(self, q1, q2, x1, x2, fit):
        eta, pi = self.eta, math.pi
        self.sig = [fit["sigma%d" % k] for k in (1, 2, 3, 4)]
        self.bet = [fit["beta%d" % k] for k in (1, 2, 3)]
        self.alp = [fit["alpha%d" % k] for k in (1, 2, 3, 4, 5)]
        SL = q1 ** 2 * x1 + q2 ** 2 * x2
        dS = (q1 - q2) * (q2 * x2 - q1 * x1)
        sigma = eta * (721.0 / 48.0 * x1 * x2 - 247.0 / 48.0 * x1 * x2)
        for q, x in ((q1, x1), (q2, x2)):
            sigma = sigma + (719.0 / 96.0 - 233.0 / 96.0) * q ** 2 * x ** 2
        gam = ((554345.0 / 1134.0 + 110.0 * eta / 9.0) * SL
               + (13915.0 / 84.0 - 10.0 * eta / 3.0) * dS)
        v = [1.0 + 0.0 * eta, 0.0 * eta, 5.0 * (743.0 / 84.0 + 11.0 * eta) / 9.0,
             -16.0 * pi + 188.0 * SL / 3.0 + 25.0 * dS,
             5.0 * (3058.673 / 7.056 + 5429.0 / 7.0 * eta + 617.0 * eta * eta) / 72.0
             - 10.0 * sigma,
             5.0 / 9.0 * (7729.0 / 84.0 - 13.0 * eta) * pi - gam,
             (11583.231236531 / 4.694215680 - 640.0 / 3.0 * pi * pi - 6848.0 / 21.0 * _EULER
              + eta * (-15737.765635 / 3.048192 + 2255.0 / 12.0 * pi * pi)
              + eta * eta * 76055.0 / 1728.0 - eta ** 3 * 127825.0 / 1296.0
              - 6848.0 / 21.0 * math.log(4.0)
              + pi * (3760.0 * SL + 1490.0 * dS) / 3.0),  # PhenomD leaves the 3PN spin-spin term out
             pi * (77096675.0 / 254016.0 + 378515.0 / 1512.0 * eta - 74045.0 / 756.0 * eta * eta)
             + (-8980424995.0 / 762048.0 + 6586595.0 * eta / 756.0 - 305.0 * eta * eta / 36.0) * SL
             - (170978035.0 / 48384.0 - 2876425.0 * eta / 672.0 - 4735.0 * eta * eta / 144.0) * dS]
        pfa = 3.0 / (128.0 * eta)
        self.v = [pfa * c for c in v]
        self.log5 = pfa * (5.0 / 3.0 * (7729.0 / 84.0 - 13.0 * eta) * pi - 3.0 * gam)
        self.log6 = pfa * (-6848.0 / 21.0)
        fj = _PHI_JOIN + 0.0 * eta
        self.c2i = self._dphi_ins(fj) - self._dphi_int(fj)
        self.c1i = self._phi_ins(fj) - self._phi_int(fj) - self.c2i * fj
        self.join = fm = 0.5 * self.rd
        self.c2m = self.c2i + self._dphi_int(fm) - self._dphi_mrd(fm)
        self.c1m = self._phi_int(fm) + self.c1i + self.c2i * fm - self._phi_mrd(fm) - self.c2m * fm

    def _amp_mrd(self, f):
        s, x = self.dm * self.g3, f - self.rd
        return torch.exp(-x * self.g2 / s) * (s * self.g1) / (x * x + s * s)

    def amp(self, f):
        t = f ** (1.0 / 3.0)
        a = self.ains
        ins = (1.0 + t ** 2 * a[0] + f * a[1] + t ** 4 * a[2] + t ** 5 * a[3] + f ** 2 * a[4]
               + t ** 7 * a[5] + t ** 8 * a[6] + f ** 3 * a[7])
        x = (f - _AMP_JOIN) / self.width
        c = self.mid
        mid = c[0] + x * (c[1] + x * (c[2] + x * (c[3] + x * c[4])))
        out = torch.where(f < _AMP_JOIN, ins, torch.where(f >= self.peak, self._amp_mrd(f), mid))
        return self.amp0 * f ** (-7.0 / 6.0) * out

    def _phi_ins(self, f):
        v, pi, t = self.v, math.pi, f ** (1.0 / 3.0)
        w = t * pi ** (1.0 / 3.0)
        logw = torch.log(w)
        s1, s2, s3, s4 = self.sig
        return (v[5] - 0.25 * pi + v[7] * w ** 2 + v[6] * w + self.log6 * logw * w
                + self.log5 * logw + v[4] / w + v[3] / w ** 2 + v[2] / w ** 3 + v[0] / w ** 5
                + (s1 * f + s2 * 0.75 * t ** 4 + s3 * 0.6 * t ** 5 + s4 * 0.5 * f ** 2) / self.eta)

    def _dphi_ins(self, f):
        v, pi, t = self.v, math.pi, f ** (1.0 / 3.0)
        w = t * pi ** (1.0 / 3.0)
        s1, s2, s3, s4 = self.sig
        s = (2.0 * v[7] * w ** 7 + (v[6] + self.log6 * (1.0 + torch.log(w))) * w ** 6
             + self.log5 * w ** 5 - v[4] * w ** 4 - 2.0 * v[3] * w ** 3 - 3.0 * v[2] * w ** 2
             - 5.0 * v[0])
        return s * pi / (3.0 * w ** 8) + (s1 + s2 * t + s3 * t ** 2 + s4 * f) / self.eta

    def _phi_int(self, f):
        b1, b2, b3 = self.bet
        return (b1 * f - b3 / (3.0 * f ** 3) + b2 * torch.log(f)) / self.eta

    def _dphi_int(self, f):
        b1, b2, b3 = self.bet
        return (b1 + b3 / f ** 4 + b2 / f) / self.eta

    def _phi_mrd(self, f):
        a1, a2, a3, a4, a5 = self.alp
        return (-a2 / f + 4.0 / 3.0 * a3 * f ** 0.75 + a1 * f + a4 * self.rho * torch.atan(
            (f - a5 * self.rd) / (self.rho * self.dm * self.tau))) / self.eta

    def _dphi_mrd(self, f):
        a1, a2, a3, a4, a5 = self.alp
        x = (f - a5 * self.rd) / (self.dm * self.tau * self.rho)
        return (a1 + a2 / f ** 2 + a3 / f ** 0.25
                + a4 / (self.dm * self.tau * (1.0 + x * x))) / self.eta

    def _pieces(self, f, ins, mid, mrd):
        return torch.where(f < _PHI_JOIN, ins, torch.where(f >= self.join, mrd, mid))

    def phase(self, f):
        return self._pieces(f, self._phi_ins(f), self._phi_int(f) + self.c1i + self.c2i * f,
                            self._phi_mrd(f) + self.c1m + self.c2m * f)

    def dphase(self, f):
        return self._pieces(f, self._dphi_ins(f), self._dphi_int(f) + self.c2i,
                            self._dphi_mrd(f) + self.c2m)


def _remnant(m1, m2, x1, x2):
    """Mass and spin of the remnant (Husa et al. 2016)."""
    q1, q2 = m1 / (m1 + m2), m2 / (m1 + m2)
    eta = q1 * q2
    s = q1 ** 2 * x1 + q2 ** 2 * x2
    spin = (3.4641016151377544 * eta - 4.399247300629289 * eta ** 2 + 9.397292189321194 * eta ** 3
            - 13.180949901606242 * eta ** 4
            + (1 - 0.0850917821418767 * eta - 5.837029316602263 * eta ** 2) * s
            + (0.1014665242971878 * eta - 2.0967746996832157 * eta ** 2) * s ** 2
            + (-1.3546806617824356 * eta + 4.108962025369336 * eta ** 2) * s ** 3
            + (-0.8676969352555539 * eta + 2.064046835273906 * eta ** 2) * s ** 4)
    s = s / (q1 ** 2 + q2 ** 2)
    erad = ((0.055974469826360077 * eta + 0.5809510763115132 * eta ** 2
             - 0.9606726679372312 * eta ** 3 + 3.352411249771192 * eta ** 4)
            * (1.0 + (-0.0030302335878845507 - 2.0066110851351073 * eta
                      + 7.7050567802399215 * eta ** 2) * s)
            / (1.0 + (-0.6714403054720589 - 1.4756929437702908 * eta
                      + 7.304676214885011 * eta ** 2) * s))
    return 1.0 - erad, spin


def _qnm(spin, mass, ell, mm):
    shift, base, amps, phases = _QNM[(ell, mm)]
    kappa = (torch.log(2.0 - spin) / math.log(3.0)) ** (1.0 / (2.0 + ell - mm))
    re = sum(a * math.cos(p) * kappa ** (k + shift) for k, (a, p) in enumerate(zip(amps, phases)))
    im = sum(a * math.sin(p) * kappa ** (k + shift) for k, (a, p) in enumerate(zip(amps, phases)))
    return (base + re) / (2.0 * math.pi * mass), im / (2.0 * math.pi * mass)


_qnm_table = []


def _qnm_22(spin, mass):
    """The tabulated (2, 2) ringdown and damping frequency that PhenomD was built with."""
    if not _qnm_table:
        from bbhx_b200.waveforms import ringdownphenomd as table

        x = _tensor(table.QNMData_a)
        y = torch.stack([_tensor(table.QNMData_fring), _tensor(table.QNMData_fdamp)])
        _qnm_table.extend([table.dspin, [c[:, 0] for c in _cubic(x[None], y[:, None])]])
    step, c = _qnm_table
    k = torch.floor((spin.detach() + 1.0) / step)
    u = spin - (step * k - 1.0)
    k = k.long()
    return [(c[0][j][k] + u * (c[1][j][k] + u * (c[2][j][k] + u * c[3][j][k]))) / mass
            for j in (0, 1)]


class _Source:
    """PhenomHM and the response of binaries P [12, B] in the given modes; arrays [B, M, L]."""

    def __init__(self, P, modes, tobs, tdi="AET"):
        self.modes, self.tdi = modes, tdi
        swap = P[0] < P[1]
        pick = lambda i, j: torch.where(swap, P[j], P[i])[:, None, None]  # noqa: E731
        m1, m2, x1, x2 = pick(0, 1), pick(1, 0), pick(2, 3), pick(3, 2)
        self.dist, self.phi, self.inc, self.lam, self.beta, self.psi, self.tref = (
            P[k][:, None, None] for k in (4, 5, 7, 8, 9, 10, 11))
        self.m1, self.m2, self.x1, self.x2 = m1, m2, x1, x2
        mass, spin = _remnant(m1, m2, x1, x2)
        rd22, dm22 = _qnm(spin, mass, 2, 2)
        lm = [_qnm(spin, mass, ell, mm) for ell, mm in modes]
        self.rdlm, dmlm = (torch.cat([z[j] for z in lm], dim=1) for j in (0, 1))
        self.rd22 = rd22
        rd, dm = _qnm_22(spin, mass)
        one = torch.ones_like(rd)
        d22 = _PhenomD(m1, m2, x1, x2, rd, dm, one, one)
        self.rho = rd22 / self.rdlm
        self.d = _PhenomD(m1, m2, x1, x2, rd, dm, self.rho, dmlm / dm22)
        self.fref = d22.peak
        self.phi0, self.t0 = 0.5 * d22.phase(self.fref), d22.dphase(self.fref)
        self.sec = (m1 + m2) * _MTSUN
        self.scale = (m1 + m2) ** 2 * _MRSUN * _MTSUN / self.dist
        self.mm = _tensor([mm for _, mm in modes])[None, :, None]
        lamb, beta = self.lam[:, 0, 0], self.beta[:, 0, 0]
        self.ts, self.te = (self._ssb(t, lamb, beta) for t in (0.0, tobs * YEAR))

    @staticmethod
    def _ssb(t, lam, beta):
        phase, rc = _OMEGA_FRAME * t - lam, _AU / _C * torch.cos(beta)
        return t + rc * torch.cos(phase) - 0.5 * _OMEGA_FRAME * rc ** 2 * torch.sin(2.0 * phase)

    def _map(self, join, trd):
        """Edges and linear pieces of the map of a mode's frequency to the (2, 2) one."""
        fi, fr = join / self.rho, self.rdlm
        ti = 2.0 * fi / self.mm
        a = (trd - ti) / (fr - fi)
        return fi, fr, a, ti - fi * a

    def phase_tf(self, f):
        Mf, d = f * self.sec, self.d
        fi, fr, a, b = self._map(_PHI_JOIN, self.rho * self.rdlm)
        low, ai = Mf <= fi, 2.0 / self.mm
        mid = ~low & (Mf <= fr)
        x = torch.where(low, ai * Mf, torch.where(mid, a * Mf + b, self.rho * Mf))
        B = d.phase(a * fi + b) / a
        A = d.phase(ai * fi) / ai
        C = d.phase(self.rho * fr) / self.rho
        D = d.phase(a * fr + b) / a - B + A
        ph = d.phase(x)
        ph = torch.where(low, ph / ai, torch.where(mid, ph / a - B + A, ph / self.rho - C + D))
        shift = _tensor([_SHIFT[mm] for _, mm in self.modes])[None, :, None]
        phase = -self.t0 * (Mf - self.fref) + shift + ph - self.mm * self.phi0
        tf = self.sec * (d.dphase(x) - self.t0) / (2.0 * math.pi)
        return phase + 2.0 * math.pi * f * self.tref, tf + self.tref

    def amp(self, f):
        Mf = f * self.sec
        fi, fr, a, b = self._map(_AMP_JOIN, self.rd22 + 0.0 * self.rdlm)
        x = torch.where(Mf > fi, torch.where(Mf > fr, Mf - self.rdlm + self.rd22, a * Mf + b),
                        2.0 / self.mm * Mf)
        ratio = []
        for i, (ell, mm) in enumerate(self.modes):
            if (ell, mm) == (2, 2):
                ratio.append(torch.ones_like(Mf[:, i]))
                continue
            h = lambda y: self._pn(ell, mm, (2.0 * math.pi / mm * y) ** (1.0 / 3.0))  # noqa: E731
            ratio.append(h(Mf[:, i]) * h(x[:, i]) / h(2.0 * Mf[:, i] / mm))
        return self.d.amp(x) * torch.stack(ratio, dim=1) * self.scale

    def _pn(self, ell, mm, v):
        q1 = (self.m1 / (self.m1 + self.m2))[:, 0]
        eta, delta = q1 * (1.0 - q1), 2.0 * q1 - 1.0
        xs, xa = 0.5 * (self.x1 + self.x2)[:, 0], 0.5 * (self.x1 - self.x2)[:, 0]
        if (ell, mm) == (2, 1):
            re = (v * delta - v ** 2 * 1.5 * (xa + delta * xs)
                  + v ** 3 * delta * (335.0 / 672.0 + eta * 117.0 / 56.0)
                  + v ** 4 * (xa * (3427.0 / 1344 - eta * 2101.0 / 336)
                              + delta * xs * (3427.0 / 1344 - eta * 965 / 336) - delta * math.pi))
            im = v ** 4 * delta * (-0.5 - 2.0 * 0.69314718056)
            return math.sqrt(2.0) / 3.0 * torch.sqrt(re ** 2 + im ** 2)
        return {(3, 3): 0.75 * math.sqrt(5 / 7) * v * delta,
                (3, 2): math.sqrt(5 / 7) / 3.0 * v ** 2 * (1.0 - 3.0 * eta),
                (4, 4): 4.0 / 9.0 * math.sqrt(10 / 7) * v ** 2 * (1.0 - 3.0 * eta),
                (4, 3): 0.75 * math.sqrt(3 / 35) * v ** 3 * delta * (1.0 - 2.0 * eta)}[(ell, mm)]

    def _harmonics(self):
        """Plus and cross weights of every mode, [B, M, 1] complex."""
        i, ct = self.inc, torch.cos(self.inc)
        c, s = torch.cos(0.5 * i), torch.sin(0.5 * i)
        pi = math.pi
        table = {
            (2, -2): math.sqrt(5 / (64 * pi)) * (1 - ct) ** 2,
            (2, -1): math.sqrt(5 / (16 * pi)) * torch.sin(i) * (1 - ct),
            (2, 1): math.sqrt(5 / (16 * pi)) * torch.sin(i) * (1 + ct),
            (2, 2): math.sqrt(5 / (64 * pi)) * (1 + ct) ** 2,
            (3, -3): math.sqrt(21 / (2 * pi)) * c * s ** 5,
            (3, -2): math.sqrt(7 / (4 * pi)) * (2 + 3 * ct) * s ** 4,
            (3, 2): math.sqrt(7 / pi) * c ** 4 * (-2 + 3 * ct) / 2,
            (3, 3): -math.sqrt(21 / (2 * pi)) * c ** 5 * s,
            (4, -4): 3 * math.sqrt(7 / pi) * c ** 2 * s ** 6,
            (4, -3): 3 * math.sqrt(7 / (2 * pi)) * c * (1 + 2 * ct) * s ** 5,
            (4, 3): -3 * math.sqrt(7 / (2 * pi)) * c ** 5 * (-1 + 2 * ct) * s,
            (4, 4): 3 * math.sqrt(7 / pi) * c ** 6 * s ** 2}
        plus, cross = [], []
        for ell, mm in self.modes:
            rot = torch.exp(1j * mm * self.phi)
            y, ym = table[(ell, mm)] * rot, (-1) ** ell * table[(ell, -mm)] * rot
            plus.append(0.5 * (y + ym))
            cross.append(0.5j * (y - ym))
        return torch.cat(plus, dim=1), torch.cat(cross, dim=1)

    def _orbit(self, t):
        """Positions of the three spacecraft and directions of the links 12, 23, 31 at t, from
        tables every 1e4 s, linear in between (Rubbo, Cornish & Poujade 2004, eq. 57)."""
        dt = 1.0e4
        w = torch.floor(t.detach() / dt)
        frac = (t - w * dt) / dt
        ends = []
        for k in (w, w + 1.0):
            al, e = _OMEGA_ORBIT * (k * dt), _ARM / (2.0 * math.sqrt(3.0) * _AU)
            ca, sa = torch.cos(al), torch.sin(al)
            x = []
            for j in range(3):
                b = 2.0 * math.pi * j / 3.0
                cb, sb = math.cos(b), math.sin(b)
                x.append(torch.stack([
                    _AU * ca + _AU * e * (sa * ca * sb - (1.0 + sa * sa) * cb),
                    _AU * sa + _AU * e * (sa * ca * cb - (1.0 + ca * ca) * sb),
                    -math.sqrt(3.0) * _AU * e * torch.cos(al - b)]))
            n = [x[i] - x[j] for i, j in ((0, 1), (1, 2), (2, 0))]
            ends.append(x + [v / torch.sqrt((v * v).sum(0)) for v in n])
        return [lo + (hi - lo) * frac for lo, hi in zip(*ends)]

    def response(self, f, t):
        """The three TDI transfers and the Roemer phase at f, t [B, M, L]."""
        cl, sl, cb, sb = (g(v) for v in (self.lam, self.beta) for g in (torch.cos, torch.sin))
        cp, sp = torch.cos(self.psi), torch.sin(self.psi)
        k = torch.stack([-cb * cl, -cb * sl, -sb])
        u = torch.stack([cp * sl - cl * sb * sp, -cl * cp - sb * sl * sp, cb * sp])
        v = torch.stack([-cl * cp * sb - sl * sp, -cp * sb * sl + cl * sp, cb * cp])
        yp, yc = self._harmonics()
        al = _OMEGA_ORBIT * t
        roemer = 2.0 * math.pi / _C * f * _AU * (k[0] * torch.cos(al) + k[1] * torch.sin(al))
        p1, p2, p3, n12, n23, n31 = self._orbit(t)
        x = math.pi * f * _ARM / _C

        def pair(n, pa, pb):
            a, b, kn = (n * u).sum(0), (n * v).sum(0), (n * k).sum(0)
            kp = (k * (pa + pb)).sum(0)
            common = 1j * x * (yp * (a * a - b * b) + yc * (2.0 * a * b)) * torch.exp(
                1j * x * (1.0 + kp / _ARM))
            sinc = lambda y: torch.where(y == 0.0, 1.0, torch.sin(y) / y)  # noqa: E731
            return common * sinc(x * (1.0 - kn)), common * sinc(x * (1.0 + kn))

        g12, g21 = pair(n31, p1, p2)
        g23, g32 = pair(n12, p2, p3)
        g31, g13 = pair(n23, p3, p1)
        z, s2 = torch.exp(2j * x), torch.sin(2.0 * x)
        if self.tdi == "XYZ":
            fac = 2j * s2 * z
            T = [fac * (g21 + z * g12 - g31 - z * g13), fac * (g32 + z * g23 - g12 - z * g21),
                 fac * (g13 + z * g31 - g23 - z * g32)]
            return T, roemer
        fae = 1j * math.sqrt(2.0) * s2 * z
        ft = 2.0 * math.sqrt(2.0) * s2 * torch.sin(x) * torch.exp(3j * x)
        f2 = -4j * torch.sin(4.0 * x) * torch.exp(4j * x)
        A = 0.5 * ((1.0 + z) * (g31 + g13) - g23 - z * g32 - g21 - z * g12)
        E = 0.5 / math.sqrt(3.0) * ((1.0 - z) * (g13 - g31) + (2.0 + z) * (g12 - g32)
                                    + (1.0 + 2.0 * z) * (g21 - g23))
        T = (g21 - g12 + g32 - g23 + g13 - g31) / math.sqrt(6.0)
        return [f2 * fae * A, f2 * fae * E, f2 * ft * T], roemer

    def quantities(self, f):
        """Amplitude, phase, t(f) and the parts of the three transfers, [9, B, M, L]."""
        phase, tf = self.phase_tf(f)
        T, roemer = self.response(f, tf)
        parts = [p for z in T for p in (z.real, z.imag)]
        return torch.stack([self.amp(f), phase + roemer, tf] + parts)

    def combine(self, q):
        """Modes summed, outside the observation zero: conj(T A e^(i phase)), [B, 3, L]."""
        ts, te = self.ts[:, None, None], self.te[:, None, None]
        wave = torch.where((q[2] >= ts) & (q[2] <= te), q[0], 0.0) * torch.exp(1j * q[1])
        return torch.stack([torch.conj(torch.complex(q[3 + 2 * c], q[4 + 2 * c]) * wave).sum(1)
                            for c in range(3)], dim=1)

    def templates(self, f):
        """[B, 3, L] on the frequencies f [L]."""
        return self.combine(self.quantities(f[None, None, :].expand(len(self.dist),
                                                                    len(self.modes), -1)))

    def knots(self, length):
        """Log-spaced knots over the frequencies at which a mode is observed."""
        r = torch.arange(length, dtype=torch.float64, device="cuda") / (length - 1)
        grid = 10.0 ** (math.log10(1e-4) + r * (math.log10(0.6) - math.log10(1e-4)))
        f = grid / self.sec * self.mm / 2.0
        _, tf = self.phase_tf(f)

        def cross(level, end):
            up = (tf[..., :-1] < level) & (level < tf[..., 1:])
            k = torch.argmax(up.to(torch.int8), dim=-1, keepdim=True)
            fa, fb, ta, tb = (torch.gather(v, -1, k + j) for v in (f, tf) for j in (0, 1))
            return torch.where(up.any(-1, keepdim=True),
                               (fb - fa) / (tb - ta) * (level - ta) + fa, end)

        span = (self.te - self.ts)[:, None, None]
        lo, hi = cross(0.0 * span, f[..., :1]), cross(span, f[..., -1:])
        return lo ** (1.0 - r) * hi ** r


def _template(P, modes, tobs, length, f, tdi="AET"):
    """The splined template of one binary P [12, 1] on the data grid f: first bin and [3, n]."""
    src = _Source(P, modes, tobs, tdi)
    x = src.knots(length)
    c = _cubic(x[0], src.quantities(x)[:, 0])
    lo, hi = (torch.searchsorted(f, v.detach().reshape(1), right=True).item()
              for v in (x.min(), x.max()))
    g = f[lo:hi]
    seg = torch.searchsorted(x[0].detach(), g[None].expand(len(modes), -1).contiguous(),
                             right=True) - 1
    inside = (seg >= 0) & (seg < length - 1)
    k = seg.clamp(0, length - 2)
    u = g - torch.gather(x[0], 1, k)
    c = [torch.gather(v, 2, k.expand(9, -1, -1)) for v in c]
    q = c[0] + u * (c[1] + u * (c[2] + u * c[3]))
    q = torch.cat([torch.where(inside, q[:1], 0.0), q[1:]])
    return lo, src.combine(q[:, None])[0]


def _direct(case, x):
    """<d|h>, <h|h> and, for the gradient, d lnL / d theta of every binary."""
    f, modes = _tensor(x["f"]), _mode_list(case) or ALL_MODES
    psd, data = _tensor(x["psd"]), x["data"]
    d = torch.zeros_like(f)
    d[1:] = f[1:] - f[:-1]
    d[0] = d[1]
    w2 = d / psd
    dd = (4.0 * w2 * (data.real ** 2 + data.imag ** 2)).sum()
    grad = case["kind"] == "lnl_grad"
    rows = []
    for b in range(case["batch"]):
        P = _tensor(x["params"][:, b:b + 1]).requires_grad_(grad)
        with torch.set_grad_enabled(grad):
            lo, h = _template(P, modes, case["tobs"], case["length"], f)
            band = slice(lo, lo + h.shape[1])
            dh = 4.0 * (w2[:, band] * data[:, band].conj() * h).sum()
            hh = 4.0 * (w2[:, band] * (h.real ** 2 + h.imag ** 2)).sum()
            lnl = -0.5 * (dd + hh - 2.0 * dh.real)
            g = torch.autograd.grad(lnl, P)[0][GRAD_ROWS, 0] if grad else None
        rows.append((lnl.detach(), dh.detach(), hh.detach(), g))
    lnl, dh, hh, g = zip(*rows)
    if grad:
        return {"lnl": torch.stack(lnl), "grad": torch.stack(g)}
    return {"lnl": torch.stack(lnl).cpu().numpy(), "d_h": torch.stack(dh),
            "h_h": torch.stack(hh).to(torch.complex128)}


def _heterodyned(case, x):
    """Relative binning about the injection (Cornish 2010; Zackay et al. 2018)."""
    f, tobs, L = _tensor(x["f"]), case["tobs"], case["length"]
    center = _tensor(x["injection"])
    src = _Source(center, ALL_MODES, tobs)
    probe = _tensor(np.logspace(np.log10(x["f"][0] * 0.999999999999),
                                np.log10(x["f"][-1] * 1.000000000001), L))
    band = probe[src.templates(probe)[0, 0].abs() != 0.0].cpu().numpy()
    freqs = _tensor(np.logspace(np.log10(band[0]), np.log10(band[-1]), L))
    i0 = int(torch.searchsorted(f, freqs[0]))
    i1 = int(torch.searchsorted(f, freqs[-1], right=True))
    f, data, psd = f[i0:i1], x["data"][:, i0:i1], _tensor(x["psd"])[:, i0:i1]
    h0 = x["template"][:, i0:i1]
    df = f[1] - f[0]
    bins = torch.searchsorted(freqs, f, right=True)  # the slot after the bin's lower edge
    a0 = 4.0 * h0.conj() * data / psd * df
    b0 = (4.0 * (h0.real ** 2 + h0.imag ** 2) / psd * df).to(torch.complex128)
    off = f - 0.5 * (freqs[(bins - 1).clamp(max=L - 2)] + freqs[bins.clamp(max=L - 1)])
    keep = slice(0, len(f) - 1)
    K = [torch.zeros((3, L), dtype=torch.complex128, device="cuda").index_add_(
        1, bins[keep], v[:, keep]) for v in (a0, a0 * off, b0, b0 * off)]
    dd = (4.0 * (data.real ** 2 + data.imag ** 2) / psd * df).sum()
    ref = src.templates(freqs)
    step = freqs[1:] - freqs[:-1]
    grad = case["kind"] == "het_grad"
    rows = []
    for b in range(0, case["batch"], 1024):
        P = _tensor(x["params"][:, b:b + 1024]).requires_grad_(grad)
        with torch.set_grad_enabled(grad):
            r = _Source(P, ALL_MODES, tobs).templates(freqs) / ref
            r1 = (r[..., 1:] - r[..., :-1]) / step
            r0 = r[..., 1:] - r1 * (0.5 * step)
            dh = (K[0][:, 1:] * r0.conj() + K[1][:, 1:] * r1.conj()).sum((1, 2))
            hh = (K[2][:, 1:] * (r0.real ** 2 + r0.imag ** 2)
                  + 2.0 * K[3][:, 1:] * (r0.real * r1.real + r0.imag * r1.imag)).sum((1, 2))
            lnl = -0.5 * (dd + hh.real - 2.0 * dh.real)
            g = torch.autograd.grad(lnl.sum(), P)[0][GRAD_ROWS].T if grad else None
        rows.append((lnl.detach(), dh.detach(), hh.detach(), g))
    lnl, dh, hh, g = zip(*rows)
    if grad:
        return {"lnl": torch.cat(lnl), "grad": torch.cat(g)}
    return {"lnl": torch.cat(lnl).cpu().numpy(), "d_h": torch.cat(dh), "h_h": torch.cat(hh)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "lnl" and case["batch"] * case["tobs"] > 250.0:
        return None  # about 20 ms for each binary and year of data
    x = _inputs(case, seed)
    modes = _mode_list(case) or ALL_MODES
    if kind == "sparse":
        return torch.cat([_Source(_tensor(x["params"][:, b:b + 64]), modes, case["tobs"],
                                  case["tdi"]).templates(_tensor(_sparse_grid(case)))
                          for b in range(0, case["batch"], 64)])
    f = _tensor(x["f"])
    if kind == "fill":
        out = torch.zeros((3, len(f)), dtype=torch.complex128, device="cuda")
        for b in range(case["batch"]):
            lo, h = _template(_tensor(x["params"][:, b:b + 1]), modes, case["tobs"],
                              case["length"], f, case["tdi"])
            out[:, lo:lo + h.shape[1]] += h
        return out
    lo, h = _template(_tensor(x["injection"]), ALL_MODES, case["tobs"], 1024, f)
    x["template"] = torch.zeros((3, len(f)), dtype=torch.complex128, device="cuda")
    x["template"][:, lo:lo + h.shape[1]] = h
    x["data"] = x["noise"] + x["template"]
    return _direct(case, x) if kind in ("lnl", "lnl_grad") else _heterodyned(case, x)
