#!/usr/bin/env python
"""Benchmark of the batched BBHx waveform -> likelihood path on B200.

Workload (one "step"): the direct log-likelihood of B = 1024 massive-black-hole binaries
(seeded draws: total mass log-U[1e5, 1e7] Msun, q ~ U[0.1, 1], spins U[-0.9, 0.9], ...),
PhenomHM with 6 modes on 1024-point sparse grids, 2nd-generation TDI A/E/T, Tobs = 1 yr,
data grid df = 1/Tobs over [1e-5, 0.1] Hz (~3.16e6 bins; complex128 data and real noise
weights, ~250 MB, larger than L2), synthetic data = seeded injection + Gaussian noise from
the analytic PSD with the equal-arm TDI noise zeros notched (f = k c / 4L, +-16 bins).
Headline arithmetic: plain FP64 (the parity form); the mixed form (FP64 phase, t(f), products
and sums; FP32 amplitude and transfer) is timed beside it with its |dlnL| against FP64.

  value  : FP64 lnL evaluations / s with parameters already resident on the GPU
  e2e    : the same through the public API (Likelihood.get_ll) from pinned host params,
           including the H2D copy of the 12 x B parameters and the D2H copy of the B lnL
  roofline: the fused FP64 interpolate + reduce kernel against the FP64 pipe, with the 70
           instructions per (binary, data bin) it cannot do without; its 72 B of data and weights
           per pair against measured HBM bandwidth (`hbm`) are no bound: they are L2-resident
  cpu_baseline: the reference's own C++ CPU path (oracle/_ref) on a bounded sample

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
For N > 1 launch under torchrun; every rank evaluates its own batch (weak scaling) and the
time is the max over ranks.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)

TOBS = 1.0
F_LO, F_HI = 1e-5, 0.1
LENGTH = 1024
SEED_PARAMS = 1234
SEED_NOISE = 99
HBM_BYTES_PER_PAIR = 72.0  # 3 x complex128 weighted data + 3 x float64 noise weights
MIXED_BYTES_PER_PAIR = 36.0  # 3 x complex64 + 3 x float32: the FP32 copies the mixed form reads
# FP64 instructions per (binary, bin) pair the panel form cannot do without, whatever the number of
# modes: per channel a complex polynomial of degree 7 (14) and the products with weight and data
# (8), and one carrier product for the three (4)
FP64_INSTR_PER_PAIR = 3 * (14 + 8) + 4
# the library's kernels in one direct step (ncu launch list): k_clear_flags, k_step_front,
# k_ringdown_hm, k_ringdown_d, k_phm_setup, k_default_freqs, k_phm_tf, k_tf_window,
# k_response_setup, k_phm_response, k_tf_range, k_spline, k_support, k_grid_detect,
# k_tile_segments, k_direct_panel, k_direct_fused (returns at once on uniform grids),
# k_fused_reduce, k_pack_lnl
LAUNCHES_PER_STEP = 19


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=1024)
    ap.add_argument("--no-extra", action="store_true",
                    help="skip every metric after the headline (spline, heterodyned, gradients, uneven)")
    ap.add_argument("--no-het", action="store_true", help="skip the heterodyned metric")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline")
    ap.add_argument("--het-batch", type=int, default=65536)
    ap.add_argument("--grad-batch", type=int, default=4096)
    ap.add_argument("--no-grad", action="store_true", help="skip the gradient metric")
    ap.add_argument("--no-uneven", action="store_true", help="skip the uneven-batch metric")
    ap.add_argument("--uneven-batch", type=int, default=16384)
    return ap.parse_args()


def workload_name(B, N):
    return ("direct lnL, plain FP64, B=%d binaries x 6 modes, sparse L=%d, Tobs=1 yr, "
            "df=1/Tobs over 1e-5..0.1 Hz (N=%d bins), AET TDI2" % (B, LENGTH, N))


def shard_seed(rank):
    """Seed of rank's binaries: every rank evaluates its own batch (weak scaling, no
    data-path collective; binaries are independent)."""
    return SEED_PARAMS + 1000 * rank


def max_over_ranks(value, world, device="cuda"):
    """Max of a per-rank float over all ranks (device-timed numbers use the slowest rank)."""
    if world <= 1:
        return float(value)
    import torch
    import torch.distributed as dist

    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def aggregate_rate(units_per_rank, world, ms):
    """Whole-job throughput: units processed by all ranks / the max-over-ranks time."""
    return units_per_rank * world / (ms / 1e3)


def rank_info():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)),
            int(os.environ.get("LOCAL_RANK", 0)))


# --------------------------------------------------------------------------- CPU (oracle)
def _cpu_worker(args):
    """One spawn worker: the reference CPU path (oracle/_ref) for a chunk of binaries."""
    chunk, = args
    sys.path.insert(0, REPO)
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import data_grid, gaussian_noise, notch_tdi_zeros
    from oracle.pipeline import RefPipeline

    f = data_grid(TOBS, F_LO, F_HI)
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    data = gaussian_noise(psd, f[1] - f[0], SEED_NOISE)
    pipe = RefPipeline("ref", tdi2=True)
    t0 = time.perf_counter()
    pipe.direct_lnl(chunk, f, data, psd, length=LENGTH, t_obs_end=TOBS)
    return time.perf_counter() - t0


def cpu_reference(params, workers, steps=1, warmup=0):
    """Time the reference CPU path with `workers` processes, one binary each per step.
    Returns (binaries per second, per-step seconds list)."""
    import multiprocessing as mp

    ctx = mp.get_context("spawn")
    B = params.shape[1]
    times = []
    with ctx.Pool(workers) as pool:
        for s in range(warmup + steps):
            idx = [(s * workers + w) % B for w in range(workers)]
            chunks = [(params[:, i:i + 1].copy(),) for i in idx]
            # a step is the slowest worker's lnL call (data and PSD set-up inside the worker
            # are not part of the reference's per-call work)
            dt = max(pool.map(_cpu_worker, chunks))
            if s >= warmup:
                times.append(dt)
    return workers / statistics.mean(times), times


def cpu_workers():
    n = os.cpu_count() or 1
    return max(1, min(n, 64))


# --------------------------------------------------------------------------- clocks
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        import tempfile

        fd, self.path = tempfile.mkstemp(prefix=f"bbhx_clocks_gpu{gpu_index}_", suffix=".csv")
        os.close(fd)
        self.proc = None
        try:
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200", "-i", str(gpu_index)], stdout=self.fh, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = float(parts[2])
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        try:
            os.remove(self.path)
        except OSError:
            pass
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


# --------------------------------------------------------------------------- GPU arm
def measured_peaks():
    try:
        return json.load(open(os.path.join(REPO, "MEASURED_PEAKS.json")))
    except Exception:
        return None


def ncu_traffic_per_pair():
    """DRAM bytes per (binary, bin) of the fused kernel from the committed ncu summary."""
    try:
        d = json.load(open(os.path.join(REPO, "profiles", "direct_fused_traffic.json")))
        return float(d["dram_bytes_per_pair"])
    except Exception:
        return None


def make_wave():
    from bbhx_b200 import BBHWaveformFD, EqualArmlengthOrbits

    return BBHWaveformFD(response_kwargs=dict(orbits=EqualArmlengthOrbits(), TDItag="AET", tdi2=True))


def build_problem(B, seed_params=SEED_PARAMS):
    import torch

    from bbhx_b200 import Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import data_grid, draw_params, gaussian_noise, notch_tdi_zeros

    f = data_grid(TOBS, F_LO, F_HI)
    df = f[1] - f[0]
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    wave = make_wave()
    inj = draw_params(1, TOBS, seed_params + 7)
    h = wave(*inj, freqs=f, length=LENGTH, t_obs_start=0.0, t_obs_end=TOBS, direct=False,
             fill=True, combine=True)
    data = gaussian_noise(psd, df, SEED_NOISE) + h.cpu().numpy()
    like = Likelihood(wave, f, data, psd)
    like.raw_data = data
    like.injection = inj[:, 0]
    params = draw_params(B, TOBS, seed_params)
    torch.cuda.synchronize()
    return wave, like, params, f


def gpu_arm(args):
    import torch

    rank, world, local = rank_info()
    if world > 1:
        import datetime

        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    else:
        torch.cuda.set_device(0)
    from bbhx_b200 import build_ext

    build_ext.build()
    from bbhx_b200.likelihood import pack_lnl

    B = args.batch
    wave, like, params, f = build_problem(B, shard_seed(rank))
    dev_params = tuple(torch.as_tensor(params[k], device="cuda") for k in range(12))
    kw = dict(length=LENGTH, t_obs_start=0.0, t_obs_end=TOBS)
    flags = torch.zeros(3, dtype=torch.int32, device="cuda")

    def step(timing=None, precision="fp64"):
        d_h, h_h = wave.inner_products(dev_params, like.data_freqs, like.data_channels,
                                       like.noise_factors, flags=flags, timing=timing,
                                       precision=precision,
                                       data32=like.fp32_data() if precision == "mixed" else None,
                                       **kw)
        return pack_lnl(d_h, h_h, like.d_d)

    def barrier():
        if world > 1:
            import torch.distributed as dist

            dist.barrier()

    def timed(precision, timing, sampler_on=False):
        for _ in range(args.warmup):
            step(precision=precision)
        torch.cuda.synchronize()
        barrier()
        torch.cuda.synchronize()
        sampler = ClockSampler(local) if sampler_on else None
        a = torch.cuda.Event(enable_timing=True)
        z = torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(args.steps):
            res = step(timing, precision=precision)
        z.record()
        torch.cuda.synchronize()
        barrier()
        clk = sampler.stop() if sampler else None
        return a.elapsed_time(z), res, clk

    # headline: the plain FP64 form (the parity form, results identical to the reference's
    # FP64 path within 1e-6 + 2e-11 |lnL|)
    timing = {}
    ms_total, out64, clocks = timed("fp64", timing, sampler_on=(rank == 0 or world > 1))
    if int(flags.abs().sum().item()) != 0:
        raise RuntimeError(f"device error flags set: {flags.tolist()}")
    fused_ms = [a.elapsed_time(b) for a, b in timing["fused"]]
    spline_ms = [a.elapsed_time(b) for a, b in timing["spline"]]
    ms_total = max_over_ranks(ms_total, world)
    # mixed form (FP32 amplitude / transfer) beside it, with its error against FP64
    mixed_timing = {}
    mixed_ms, outmx, _ = timed("mixed", mixed_timing)
    mixed_ms = max_over_ranks(mixed_ms, world)
    lnl64 = out64.cpu().numpy()
    lnlmx = outmx.cpu().numpy()
    assert np.all(np.isfinite(lnlmx)) and np.all(np.isfinite(lnl64)), "non-finite lnL"
    dl_mixed = np.abs(lnlmx - lnl64)
    _, hh64 = wave.inner_products(dev_params, like.data_freqs, like.data_channels,
                                  like.noise_factors, flags=flags, precision="fp64", **kw)
    hh64 = hh64.real.cpu().numpy()

    # support sizes (sum of per-binary data-grid lengths) for the roofline
    from bbhx_b200 import _lib

    x = wave._last_x
    sup = torch.zeros(2 * B, dtype=torch.int32, device="cuda")
    _lib.call("bbhx_template_support", _lib.dptr(sup), _lib.dptr(sup[B:]), _lib.dptr(x),
              wave.num_modes, LENGTH, B, _lib.dptr(like.data_freqs), len(f), _lib.stream())
    pairs = float(sup[B:].double().sum().item())

    # end to end through the public API (Likelihood.get_ll) from pinned host memory: the H2D
    # copy of the parameters and the D2H copy of the results are inside the timed region
    host = torch.tensor(params, dtype=torch.float64).pin_memory()

    def e2e(precision):
        like.precision = precision
        for _ in range(2):
            like.get_ll(host, **kw)
        torch.cuda.synchronize()
        barrier()
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record()
        for _ in range(args.steps):
            ll_host = like.get_ll(host, **kw)
        t1.record()
        torch.cuda.synchronize()
        return max_over_ranks(t0.elapsed_time(t1), world), ll_host

    e2e_ms, ll_host = e2e("fp64")
    e2e_mx_ms, _ = e2e("mixed")
    like.precision = "fp64"
    dl = float(np.max(np.abs(ll_host - lnl64)))
    near = near_peak_direct(like, kw)

    extra = {}
    # the heterodyned / gradient / uneven-batch metrics are single-GPU figures; a multi-rank run
    # reports the headline direct lnL only (every rank's own batch, no collective)
    if not args.no_extra and world == 1:
        extra.update(spline_metric(timing, B, wave.num_modes))
        if not args.no_het:
            extra.update(het_metric(args, wave, like, f, params))
        if not args.no_grad:
            extra.update(grad_metric(args))
        if not args.no_uneven:
            extra.update(uneven_metric(args))
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()
    if rank != 0:
        return None
    peaks = measured_peaks()
    peak = peaks["hbm_gbs"] if peaks else 6650.0
    fused_avg_s = statistics.mean(fused_ms) / 1e3
    achieved = HBM_BYTES_PER_PAIR * pairs / fused_avg_s / 1e9
    tpp = ncu_traffic_per_pair()
    n_evals = B * args.steps * world
    mixed_kernel_ms = statistics.mean(a.elapsed_time(b) for a, b in mixed_timing["fused"])
    res = {
        "metric": "lnL evals/s (direct, heterodyned) mixed vs FP64 plain at |dlnL|<=1e-2; grad/s",
        "value": aggregate_rate(B * args.steps, world, ms_total),
        "unit": "lnL evals/s",
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": ms_total / args.steps,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic: seeded PhenomHM injection + Gaussian noise from the analytic A/E/T PSD",
        "mixed": {"value": aggregate_rate(B * args.steps, world, mixed_ms), "unit": "lnL evals/s",
                  "ms_per_step": mixed_ms / args.steps, "kernel_ms": mixed_kernel_ms,
                  "e2e": aggregate_rate(B * args.steps, world, e2e_mx_ms),
                  "dtype": "mixed: f64 phase/t(f)/products/accumulation, f32 amplitude/transfer",
                  "dlnl_vs_fp64": {"max": float(dl_mixed.max()),
                                   "p99": float(np.percentile(dl_mixed, 99)),
                                   "median": float(np.median(dl_mixed)),
                                   "max_over_hh": float(np.max(dl_mixed / np.maximum(1.0, hh64))),
                                   "frac_within_1e-2": float(np.mean(dl_mixed <= 1e-2)),
                                   "median_hh": float(np.median(hh64)),
                                   "near_peak": near}},
        "config": {"workload": workload_name(B, len(f)),
                   "global_batch": n_evals // args.steps, "data_bins": len(f),
                   "binary_bin_pairs_per_step": pairs,
                   "l2": "inputs larger than L2: every step writes and reads 1.8 GB of sparse buffers / "
                         "spline coefficients besides the 227 MB FP64 data and weights",
                   "parallelism": f"replicas x{world} (independent binary batches per GPU)"},
        "e2e": {"value": aggregate_rate(B * args.steps, world, e2e_ms), "unit": "lnL evals/s",
                "h2d_bytes_per_step": 12 * B * 8, "d2h_bytes_per_step": 3 * B * 8 + 3 * 8,
                "path": "Likelihood.get_ll (precision='fp64') from pinned host parameters",
                "max_abs_dlnl_vs_device_path": dl},
        "roofline": {**fp64_roofline(pairs, fused_avg_s),
                     "kernel": "k_direct_panel (bbhx_direct_like_fused, precision 0)",
                     "kernel_ms": statistics.mean(fused_ms),
                     "traffic": (tpp * pairs if tpp is not None else None),
                     "hbm": {"achieved": achieved, "peak": peak, "unit": "GB/s",
                             "frac": achieved / peak,
                             "algorithmic_bytes_per_pair": HBM_BYTES_PER_PAIR,
                             "peak_source": "MEASURED_PEAKS.json hbm_gbs (of measured)"
                                            if peaks else "fallback"}},
        "gpu_launches": LAUNCHES_PER_STEP * args.steps,
        "clocks": clocks,
    }
    res.update(extra)
    return res


def spline_metric(timing, B, M):
    """Spline build (bbhx_interpolate) inside the FP64 steps: 9 B M not-a-knot systems of
    length L per call; 5 x 8 L bytes per system (x and y read, slope and c1..c3 written, the
    shared x counted once per system)."""
    ms = statistics.mean(a.elapsed_time(b) for a, b in timing["spline"])
    systems = 9 * B * M
    nbytes = 5 * 8 * LENGTH * systems
    peaks = measured_peaks()
    peak = peaks["hbm_gbs"] if peaks else 6650.0
    gbs = nbytes / (ms / 1e3) / 1e9
    return {"spline": {"solves_per_s": systems / (ms / 1e3), "systems_per_call": systems,
                       "length": LENGTH, "kernel_ms": ms, "bytes_per_system": 5 * 8 * LENGTH,
                       "achieved_gbs": gbs, "frac_of_hbm": gbs / peak,
                       "kernel": "k_spline (cyclic reduction in shared memory, 9 right-hand sides)"}}


def near_peak_direct(like, kw, n=64):
    """Mixed vs FP64 direct lnL for binaries close to the injection (the region a sampler
    spends its time in): relative 5e-6 on masses, 5e-5 on spins and angles, 0.05 s on t_ref.
    There d - h is noise-level, so the FP32 error enters lnL as ~1e-7 sqrt(<h|h>) instead of
    the ~1e-7 <h|h> of templates far from the data."""
    from bbhx_b200.synthetic import perturb_params

    P = perturb_params(like.injection, n, 13, rel_mass=5e-6, abs_spin_angle=5e-5, t_ref_s=0.05)
    prev = like.precision
    out = {}
    for prec in ("fp64", "mixed"):
        like.precision = prec
        out[prec] = like.get_ll(P, **kw)
    hh = float(np.median(like.h_h.real.cpu().numpy()))
    like.precision = prev
    e = np.abs(out["mixed"] - out["fp64"])
    return {"binaries": n, "lnl_below_max": float(out["fp64"].max() - out["fp64"].min()),
            "median_hh": hh, "max": float(e.max()), "median": float(np.median(e)),
            "frac_within_1e-2": float(np.mean(e <= 1e-2))}


def het_metric(args, wave, like, f, params):
    """Heterodyned lnL evals/s: 128 relative-binning bins, B walkers around the injection.

    Three forms on the same walkers: the fused kernel in FP64 ("plain FP64 GPU form") and in
    mixed precision, and the step-by-step chain of the reference (sparse templates, ratio,
    hdyn).  |dlnL| of mixed against FP64 is reported over all walkers."""
    import torch

    from bbhx_b200 import AET1SensitivityMatrix, HeterodynedLikelihood
    from bbhx_b200.synthetic import perturb_params

    kw = dict(t_obs_start=0.0, t_obs_end=TOBS)
    center = like.injection
    data = like.raw_data
    het = HeterodynedLikelihood(wave, f, data, center, 128, template_gen_kwargs=dict(kw),
                                reference_gen_kwargs=dict(kw, length=LENGTH),
                                sens_mat=AET1SensitivityMatrix(f, tdi2=True, notch=True))
    Bh = args.het_batch
    walkers = torch.as_tensor(perturb_params(center, Bh, 5), device="cuda")
    n = max(2, args.steps // 2)

    def timed(precision, batch):
        het.precision = precision
        w = walkers[:, :batch]
        for _ in range(2):
            het.get_ll(w, **kw)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(n):
            ll = het.get_ll(w, **kw)
        e1.record()
        torch.cuda.synchronize()
        return batch * n / (e0.elapsed_time(e1) / 1e3), ll

    v64, ll64 = timed("fp64", Bh)
    vmx, llmx = timed("mixed", Bh)
    # walkers close to the reference point (where the sampler spends its time)
    wn = torch.as_tensor(perturb_params(center, 4096, 11, rel_mass=5e-6, abs_spin_angle=5e-5,
                                        t_ref_s=0.05), device="cuda")
    het.precision = "fp64"
    ln64 = het.get_ll(wn, **kw)
    het.precision = "mixed"
    lnmx = het.get_ll(wn, **kw)
    en = np.abs(lnmx - ln64)
    chain_batch = min(Bh, 16384)
    vch, _ = timed(None, chain_batch)
    d = np.abs(llmx - ll64)
    # both heterodyned forms against the direct FP64 lnL (the form pinned to the reference) on
    # the first walkers: relative-binning error plus, for mixed, the precision error.  The
    # heterodyne keeps only the data inside the reference template's band (as the reference
    # does), so its <d|d> lacks the rest: that walker-independent constant is removed first.
    nd = min(Bh, 1024)
    prev = like.precision
    like.precision = "fp64"
    ll_dir = like.get_ll(walkers[:, :nd], length=LENGTH, **kw)
    like.precision = prev
    dd_offset = 0.5 * (like.d_d - het.reference_d_d)

    def vs_direct(ll):
        e = np.abs(ll[:nd] - (ll_dir + dd_offset))
        return {"max": float(e.max()), "median": float(np.median(e)),
                "frac_within_1e-2": float(np.mean(e <= 1e-2))}
    roof = het_roofline(het, wave, center, v64)
    return {"heterodyned": {
        "value": vmx, "unit": "lnL evals/s", "batch": Bh, "bins": 128,
        "roofline_fp64": roof,
        "dtype": "mixed: f64 phase/t(f)/Roemer/ratio/sums, f32 amplitude/transfer/products",
        "fp64_plain": {"value": v64, "unit": "lnL evals/s", "kernel": "k_het_fused<fp64>"},
        "mixed_over_fp64": vmx / v64,
        "step_by_step_chain_fp64": {"value": vch, "unit": "lnL evals/s", "batch": chain_batch},
        "dlnl_mixed_vs_fp64": {"max": float(d.max()), "p99": float(np.percentile(d, 99)),
                               "median": float(np.median(d)),
                               "frac_within_1e-2": float(np.mean(d <= 1e-2)),
                               "max_over_reference_hh": float(d.max() / het.reference_h_h),
                               "reference_hh": float(het.reference_h_h),
                               "near_peak": {"walkers": 4096,
                                             "lnl_below_max": float(ln64.max() - ln64.min()),
                                             "max": float(en.max()), "median": float(np.median(en)),
                                             "frac_within_1e-2": float(np.mean(en <= 1e-2))}},
        "dlnl_vs_direct_fp64": {"walkers": nd, "dd_out_of_band_half": dd_offset,
                                "mixed": vs_direct(llmx), "fp64": vs_direct(ll64)},
        "lnl_range": [float(ll64.min()), float(ll64.max())],
        "path": "HeterodynedLikelihood.get_ll with device-resident walkers",
        "finite": bool(np.all(np.isfinite(ll64)) and np.all(np.isfinite(llmx)))}}


def fp64_lane_rate():
    """FP64 lane operations per second: the device's SMs x 64 FP64 lanes (B200) x the nominal
    1965 MHz SM clock."""
    import torch

    try:
        sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    except Exception:
        sms = 148
    return sms * 64 * 1.965e9
OPC_NAMES = ("add_sub", "mul", "div", "compare", "sqrt", "cbrt", "log", "exp", "pow", "atan",
             "sin_cos", "other")


def fp64_roofline(pairs, kernel_s):
    """The FP64 pipe's bound on the direct kernel: FP64_INSTR_PER_PAIR instructions for every pair
    (the panels' nodes and the bins evaluated one by one come on top) at the nominal FP64 lane rate
    give the shortest possible kernel time."""
    work, peak = FP64_INSTR_PER_PAIR * pairs, fp64_lane_rate()
    return {"bound": "fp64", "achieved": work / kernel_s / 1e12, "peak": peak / 1e12,
            "unit": "T FP64 instructions/s", "frac": work / kernel_s / peak,
            "fp64_instr_per_pair": FP64_INSTR_PER_PAIR, "floor_ms": work / peak * 1e3,
            "peak_source": "the device's SMs x 64 FP64 lanes x 1965 MHz (nominal clock)"}


def het_roofline(het, wave, center, evals_per_s):
    """FP64 roofline of the heterodyned form: the algorithmic operations of one (walker, mode,
    frequency) point, tallied by running the templated FP64 model on an op-counting scalar
    (bbhx_count_point_ops; the per-binary set-up and the per-bin relative-binning arithmetic
    are excluded), times the points per second, against the nominal FP64 lane rate (the
    device's SMs x 64 lanes x 1965 MHz; the measured peaks hold no FP64 figure)."""
    import torch

    from bbhx_b200 import _lib
    from bbhx_b200.waveforms.ringdownphenomd import dspin

    ap, rg = wave.amp_phase_gen, wave.response_gen
    prm = torch.tensor([center[k] for k in (0, 1, 2, 3, 4, 5, 7, 8, 9, 10, 11)],
                       dtype=torch.float64, device="cuda")
    out = torch.zeros(12, dtype=torch.int64, device="cuda")
    M, L = len(ap.allowable_modes), int(het.freqs.numel())
    tab = ap.qnm_table
    _lib.call("bbhx_count_point_ops", rg.orbit_handle.ptr, _lib.dptr(out), _lib.dptr(prm),
              _lib.dptr(ap.ells_default), _lib.dptr(ap.mms_default), M, _lib.dptr(het.freqs), L,
              _lib.dptr(tab), int(tab.shape[1]), float(dspin), rg.TDItag_int, int(rg.rescaled),
              int(rg.tdi2), _lib.stream())
    tally = out.cpu().numpy() / float(M * L)
    per_point = {k: float(v) for k, v in zip(OPC_NAMES, tally)}
    arith = float(tally[0] + tally[1] + tally[2])
    special = float(tally[4:11].sum())
    points_per_s = evals_per_s * M * L
    return {"ops_per_point": per_point, "arith_ops_per_point": arith,
            "elementary_calls_per_point": special, "points_per_s": points_per_s,
            "arith_ops_per_s": arith * points_per_s, "peak_lane_ops_per_s": fp64_lane_rate(),
            "frac_arith": arith * points_per_s / fp64_lane_rate(),
            "form": "FP64 fused kernel (k_het_fused<FP64>)",
            "peak_source": "nominal (the device's SMs x 64 FP64 lanes x 1965 MHz); cross-check: ncu FP64 pipe % in profiles/"}


def grad_metric(args):
    """Gradient evals/s (d lnL / d theta, 11 parameters, FP64) and peak device memory:
    direct lnL for B = 4096 binaries at Tobs = 0.25 yr (df = 1/Tobs over 1e-5..0.1 Hz), and
    heterodyned lnL for B = 65536 walkers (128 bins) around the injection.  Each gradient call
    recomputes the waveform (nothing is kept from the lnL evaluation)."""
    import torch

    from bbhx_b200 import AET1SensitivityMatrix, HeterodynedLikelihood, Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import (data_grid, draw_params, gaussian_noise, notch_tdi_zeros,
                                     perturb_params)

    tobs = 0.25
    f = data_grid(tobs, F_LO, F_HI)
    df = f[1] - f[0]
    psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
    wave = make_wave()
    P = draw_params(args.grad_batch, tobs, SEED_PARAMS + 7)
    center = P[:, 0]
    kw = dict(t_obs_start=0.0, t_obs_end=tobs, length=LENGTH)
    inj = wave(*[np.atleast_1d(v) for v in center], freqs=f, fill=True, direct=False, **kw)[0]
    data = inj.cpu().numpy() + gaussian_noise(psd, df, SEED_NOISE + 7)
    like = Likelihood(wave, f, data, psd)
    Pd = torch.as_tensor(P, device="cuda")

    def timed(fn, n):
        fn()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(n):
            out = fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / 1e3 / n, torch.cuda.max_memory_allocated() / 1e9, out

    sd, memd, (_, gd) = timed(lambda: like.get_ll_and_grad(Pd, **kw), 2)
    het = HeterodynedLikelihood(wave, f, data, center, 128,
                                template_gen_kwargs=dict(t_obs_start=0.0, t_obs_end=tobs),
                                reference_gen_kwargs=dict(kw),
                                sens_mat=AET1SensitivityMatrix(f, tdi2=True, notch=True))
    W = torch.as_tensor(perturb_params(center, args.het_batch, 3), device="cuda")
    sh, memh, (_, gh) = timed(lambda: het.get_ll_and_grad(W, t_obs_start=0.0, t_obs_end=tobs), 3)
    return {"gradients": {
        "direct": {"value": args.grad_batch / sd, "unit": "grad evals/s", "batch": args.grad_batch,
                   "data_bins": int(len(f)), "tobs_yr": tobs, "peak_mem_gb": memd,
                   "finite": bool(torch.isfinite(gd).all().item())},
        "heterodyned": {"value": args.het_batch / sh, "unit": "grad evals/s", "batch": args.het_batch,
                        "bins": 128, "peak_mem_gb": memh,
                        "finite": bool(torch.isfinite(gh).all().item())},
        "parameters": "m1, m2, chi1z, chi2z, distance, phi_ref, inc, lam, beta, psi, t_ref",
        "method": "adjoint of the reduction / spline chain + dual-number tangents of PhenomHM + TDI"}}


def uneven_metric(args):
    """Uneven batch: 16384 binaries mixing (2,2)-only and the 6 HM modes, sparse grids of
    256/512/1024/2048 points and observation spans of 0.1/0.5/1 yr (24 direct groups, one
    persistent launch), plus heterodyned instances with 64/128/192/256 bins (1024 walkers
    each); mixed precision, captured in a CUDA graph with the autotuned launch shape.
    Compared with the plain FP64 GPU form evaluating the same groups one call at a time."""
    import torch

    from bbhx_b200 import AET1SensitivityMatrix, HeterodynedLikelihood, Likelihood
    from bbhx_b200.sensitivity import aet_psd
    from bbhx_b200.synthetic import (data_grid, draw_params, gaussian_noise, notch_tdi_zeros,
                                     perturb_params)
    from bbhx_b200.uneven import Autotuner, DirectGroup, HetGroup, UnevenBatch
    from bbhx_b200.utils.constants import YRSID_SI

    n_total = args.uneven_batch
    tobs_list, lengths, modesets = (0.1, 0.5, 1.0), (256, 512, 1024, 2048), ([(2, 2)], None)
    ngroups = len(tobs_list) * len(lengths) * len(modesets)
    per = n_total // ngroups
    likes, direct = {}, []
    seed = SEED_PARAMS + 31
    for tobs in tobs_list:
        f = data_grid(tobs, F_LO, F_HI)
        psd = notch_tdi_zeros(f, np.array([aet_psd(f, c, tdi2=True) for c in "AET"]))
        wave = make_wave()
        inj = draw_params(1, tobs, seed)
        h = wave(*inj, freqs=f, length=LENGTH, t_obs_start=0.0, t_obs_end=tobs, direct=False,
                 fill=True, combine=True)
        data = gaussian_noise(psd, f[1] - f[0], seed) + h.cpu().numpy()
        likes[tobs] = (Likelihood(wave, f, data, psd), f, data, inj[:, 0])
        for L in lengths:
            for modes in modesets:
                seed += 1
                prm = draw_params(per, tobs, seed)
                # t_ref in [0.8, 0.95] Tobs: draws closer to the end can cross the window twice,
                # which the reference rejects (phenomhm.py:557-583)
                prm[11] = np.random.default_rng(seed).uniform(0.8, 0.95, per) * tobs * YRSID_SI
                direct.append(dict(like=likes[tobs][0], params=prm, length=L, modes=modes,
                                   tobs=tobs))
    het_groups = []
    like1, f1, data1, inj1 = likes[1.0]
    for nb in (64, 128, 192, 256):
        het = HeterodynedLikelihood(make_wave(), f1, data1, inj1, nb,
                                    template_gen_kwargs=dict(t_obs_start=0.0, t_obs_end=1.0),
                                    reference_gen_kwargs=dict(t_obs_start=0.0, t_obs_end=1.0,
                                                              length=LENGTH),
                                    sens_mat=AET1SensitivityMatrix(f1, tdi2=True, notch=True))
        het_groups.append((het, perturb_params(inj1, 1024, nb)))

    def groups():
        dg = [DirectGroup(d["like"], d["params"], length=d["length"], modes=d["modes"],
                          t_obs_start=0.0, t_obs_end=d["tobs"]) for d in direct]
        hg = [HetGroup(h, w, t_obs_start=0.0, t_obs_end=1.0) for h, w in het_groups]
        return dg, hg

    n_inst = sum(d["params"].shape[1] for d in direct) + sum(w.shape[1] for _, w in het_groups)
    dg, hg = groups()
    batch = UnevenBatch(dg, hg, precision="mixed", autotuner=Autotuner(repeats=1))
    batch.autotuner.CTAS = (2, 3, 4)
    outs = batch.capture()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    reps = 3
    e0.record()
    for _ in range(reps):
        batch.replay()
    e1.record()
    torch.cuda.synchronize()
    t_mixed = e0.elapsed_time(e1) / 1e3 / reps
    mixed = [o.cpu().numpy() for o in outs]
    flags_ok = all(int(fl.abs().sum().item()) == 0 for fl in batch.flags())
    # plain FP64 GPU form: one call per group, no graph
    ref = []
    hh = []
    torch.cuda.synchronize()
    e0.record()
    for d in direct:
        lk = d["like"]
        lk.precision = "fp64"
        ref.append(lk.get_ll(d["params"], length=d["length"], modes=d["modes"], t_obs_start=0.0,
                             t_obs_end=d["tobs"]))
        hh.append(lk.h_h.real.cpu().numpy())
    for het, w in het_groups:
        het.precision = "fp64"
        ref.append(het.get_ll(w, t_obs_start=0.0, t_obs_end=1.0))
        hh.append(het.hdyn_h_h.real.cpu().numpy())
    e1.record()
    torch.cuda.synchronize()
    t_fp64 = e0.elapsed_time(e1) / 1e3
    err = [np.abs(a - b) for a, b in zip(mixed, ref)]
    rel = [e / np.maximum(h, 1.0) for e, h in zip(err, hh)]
    allerr = np.concatenate(err)
    allrel = np.concatenate(rel)
    labels = ["direct Tobs=%g L=%d %s bins/knot=%d" % (d["tobs"], d["length"],
                                                        "22" if d["modes"] else "HM",
                                                        len(d["like"].data_freqs) // d["length"])
              for d in direct] + ["het bins=%d" % h.length_f_het for h, _ in het_groups]
    per_group = [{"group": lb, "precision": pr, "max": float(e.max()),
                  "frac_within_1e-2": float(np.mean(e <= 1e-2))}
                 for lb, pr, e in zip(labels, batch.group_precisions(), err)]
    return {"uneven": {
        "value": n_inst / t_mixed, "unit": "lnL evals/s", "instances": int(n_inst),
        "direct_groups": len(direct), "heterodyned_groups": len(het_groups),
        "fp64_plain_per_group": {"value": n_inst / t_fp64, "unit": "lnL evals/s"},
        "speedup_vs_fp64_plain": t_fp64 / t_mixed,
        "launch_shape": {pr: {"tile_bins": sh[0], "ctas_per_sm": sh[1]} for pr, sh in batch.shape.items()},
        "groups_in_fp64": sum(1 for pr in batch.group_precisions()[:len(direct)] if pr == "fp64"),
        "dlnl_mixed_vs_fp64": {"max": float(allerr.max()), "median": float(np.median(allerr)),
                               "frac_within_1e-2": float(np.mean(allerr <= 1e-2)),
                               "p99": float(np.percentile(allerr, 99)),
                               "max_over_hh": float(allrel.max()),
                               "per_group": per_group},
        "flags_clear": flags_ok,
        "config": "mode sets (2,2) / 6 HM; L 256/512/1024/2048; Tobs 0.1/0.5/1 yr; t_ref in "
                  "[0.8, 0.95] Tobs; heterodyne bins 64/128/192/256 x 1024 walkers; CUDA graph replay"}}


CPU_STEPS, CPU_WARMUP = 4, 2  # bounded sample of the GPU line's cpu_baseline leg


def cpu_baseline(args):
    """The reference CPU path on the box's host cores, timed the same way as the reference
    arm (warm-up steps first, then the mean over timed steps; each step = one binary per
    process at the full workload size), on a bounded sample: CPU_STEPS timed steps after
    CPU_WARMUP.  Also the single-thread "as shipped" figure: the reference's CPU build never
    enables OpenMP, so one binary on one core is what its own build delivers."""
    from bbhx_b200.synthetic import draw_params
    from oracle.build_ref import OUT

    if not os.path.exists(OUT):
        return {"unavailable": "the reference's CPU library is not built (oracle/build_ref.py)"}
    params = draw_params(args.batch, TOBS, SEED_PARAMS)
    workers = cpu_workers()
    val, times = cpu_reference(params, workers, steps=CPU_STEPS, warmup=CPU_WARMUP)
    val1, times1 = cpu_reference(params, 1, steps=2, warmup=1)
    return {"value": val, "unit": "lnL evals/s", "cores": workers, "kind": "reference",
            "sample": f"{CPU_STEPS} steps after {CPU_WARMUP} warm-up, {workers} binaries per step "
                      "(one per process) at the full workload size; reference C++ CPU path "
                      "(oracle/_ref) with the reference driver logic",
            "step_seconds": times,
            "single_thread_as_shipped": {"value": val1, "unit": "lnL evals/s", "cores": 1,
                                         "sample": "2 binaries after 1 warm-up, one process"}}


def reference_arm(args):
    rank, world, _ = rank_info()
    if rank != 0:
        return None
    from bbhx_b200.synthetic import data_grid
    from bbhx_b200.synthetic import draw_params
    from oracle.build_ref import OUT

    if not os.path.exists(OUT):
        return {"impl": "reference",
                "unavailable": "the reference's CPU library is not built (oracle/build_ref.py)"}
    params = draw_params(args.batch, TOBS, SEED_PARAMS)
    workers = cpu_workers()
    val, times = cpu_reference(params, workers, steps=args.steps, warmup=args.warmup)
    cpu = {"value": val, "unit": "lnL evals/s", "cores": workers, "kind": "reference",
           "sample": f"{args.steps} steps after {args.warmup} warm-up, {workers} binaries per step "
                     "(one per process) at the full workload size"}
    return {"impl": "reference", "metric": "lnL evals/s (direct, heterodyned) mixed vs FP64 plain at |dlnL|<=1e-2; grad/s",
            "value": val, "unit": "lnL evals/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * statistics.mean(times),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": workload_name(args.batch, len(data_grid(TOBS, F_LO, F_HI)))},
            "cpu_baseline": cpu,
            "e2e": {"value": val, "unit": "lnL evals/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}


def main():
    args = parse()
    if args.impl == "reference":
        res = reference_arm(args)
        if res is not None:
            print(json.dumps(res), flush=True)
        return
    rank, world, _ = rank_info()
    res = gpu_arm(args)
    if res is None:
        return
    if not args.no_cpu and world == 1:
        res["cpu_baseline"] = cpu_baseline(args)
    print(json.dumps(res), flush=True)


if __name__ == "__main__":
    main()
