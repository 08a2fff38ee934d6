"""Benchmark: DDM frames/s of the b200 core on one GB300 (replicas on N GPUs).

Workload (default ``--config large``): one stack of 4000 frames of 1024 x 1024
uint8 (seeded Brownian-spot scene with drift and Poisson noise), 200
log-spaced lags 1..3999, fft mode, float-float tier.  A step is one full
structure-function computation of the stack (spatial FFTs, temporal
autocorrelation, combination); the stack (4.2 GB) and the spectrum (34 GB) are
far larger than L2, so no flush is needed between steps.

Prints one JSON line (rank 0).  ``--impl reference`` times the CPU restatement
of the reference's FP64 core on all host cores instead (the reference's own
``cpp`` core needs its CMake build and cannot be compiled from its sources
alone).
"""

from __future__ import annotations

import argparse
import importlib.util
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

CONFIGS = {
    # name: scene in fastddm_gb300.synthetic
    "large": "CONFIG3",        # 4000 x 1024^2 uint8, 200 log lags (the headline workload)
    "medium": "CONFIG2",       # 512 x 512^2 uint16, all lags, Blackman-Harris window
    "small": "CONFIG1",        # 64 x 128^2 uint16, all lags
    "large_tall": "CONFIG3_TALL",  # profiling: the large workload's temporal kernel on 64^2 frames
    "large_wide": "CONFIG3_WIDE",  # profiling: the large workload's spatial kernels on 64 frames
    "long": "CONFIG_LONG",     # 20000 x 256^2 uint8, 200 log lags (split temporal transform)
    "batch": None,             # 96 uneven stacks in one batch call (run_batch)
    "serve": None,             # Poisson request stream through the serving loop (run_serve)
    "dft_stage": None,         # the tensor-core DFT-stage decision measurement (run_dft_stage)
}


def module_alone(name: str):
    """A plain Python module of the package (scenes, lags, FFT lengths, ranks) without the package around it,
    whose import loads the library: the reference arm runs without any of that."""
    if f"alone_{name}" not in sys.modules:
        spec = importlib.util.spec_from_file_location(f"alone_{name}", ROOT / "fastddm_gb300" / f"{name}.py")
        sys.modules[spec.name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[spec.name])
    return sys.modules[f"alone_{name}"]


def lags_for(name: str, T: int) -> np.ndarray:
    lg = module_alone("lags")
    if name in ("large", "large_tall", "long"):
        return np.unique(lg.logspace_int(T - 1, num=200, endpoint=True))
    return np.arange(1, T)


def workload_desc(name, scene, lags, precision, mode):
    return {
        "workload": f"ddm_{mode}_{scene.length}x{scene.height}x{scene.width}_{scene.dtype}_{len(lags)}lags",
        "frames": scene.length, "height": scene.height, "width": scene.width, "pixel_dtype": scene.dtype,
        "lags": int(len(lags)), "mode": mode, "precision": precision,
        "window": "blackman_harris" if name == "medium" else None,
        "scene": {"spots": scene.n_spots, "sigma": scene.sigma, "amplitude": scene.amplitude,
                  "diffusivity": scene.diffusivity, "offset": scene.offset, "drift": scene.drift,
                  "seed": scene.seed},
        "l2_flush": "inputs larger than L2 (stack and spectrum > 129 MB)",
        "parallelism": "replicas",
    }


# ---------------------------------------------------------------------------
# CPU sample work (the oracle port); module-level so a spawn pool can run it
# ---------------------------------------------------------------------------
def _cpu_spatial(args):
    frames, nx, ny = args
    sys.path.insert(0, str(ROOT / "oracle"))
    import ddm_oracle as oracle

    t0 = time.perf_counter()
    oracle.spatial_fft(frames, nx, ny, None)
    return time.perf_counter() - t0, frames.shape[0]


def _cpu_temporal(args):
    """Temporal stage of the oracle on `nq` spectrum columns, in blocks of 2048 columns."""
    T, nq, lags, nt, seed = args
    sys.path.insert(0, str(ROOT / "oracle"))
    import ddm_oracle as oracle

    rng = np.random.default_rng(seed)
    blk = min(nq, 2048)
    Fq = rng.standard_normal((T, blk)) + 1j * rng.standard_normal((T, blk))
    t0 = time.perf_counter()
    done = 0
    while done < nq:
        n = min(blk, nq - done)
        oracle.temporal_fft(Fq[:, :n], lags, nt)
        done += n
    return time.perf_counter() - t0, nq


def cpu_throughput(frames_sample: np.ndarray, T: int, Q: int, nx: int, ny: int, nt: int, lags, workers: int,
                   spatial_frames: int, temporal_q: int, pool=None) -> dict:
    """Frames/s of the full job estimated from timed samples of both stages.

    Spatial stage: `spatial_frames` frames per worker; temporal stage:
    `temporal_q` spectrum columns of length T per worker, all workers at once.
    The job's time is extrapolated from the two measured rates as
    T / spatial rate + Q / temporal rate (both stages scale linearly in their
    units); frames/s = T / that time.  Returns the rate, the wall time of the
    sample actually run and the fractions of the job it covered.
    """
    sp_args = [(frames_sample[:spatial_frames], nx, ny) for _ in range(workers)]
    tq_args = [(T, temporal_q, list(lags), nt, i) for i in range(workers)]
    if pool is None:
        sp = [_cpu_spatial(a) for a in sp_args[:1]]  # warm-up (imports, FFT plans)
        t0 = time.perf_counter()
        sp = [_cpu_spatial(a) for a in sp_args]
        sp_wall = time.perf_counter() - t0
        t0 = time.perf_counter()
        tq = [_cpu_temporal(a) for a in tq_args]
        tq_wall = time.perf_counter() - t0
    else:
        t0 = time.perf_counter()
        sp = list(pool.map(_cpu_spatial, sp_args))
        sp_wall = time.perf_counter() - t0
        t0 = time.perf_counter()
        tq = list(pool.map(_cpu_temporal, tq_args))
        tq_wall = time.perf_counter() - t0
    nframes = sum(n for _, n in sp)
    nmodes = sum(n for _, n in tq)
    job = T * sp_wall / nframes + Q * tq_wall / nmodes
    return {"value": T / job, "sample_s": sp_wall + tq_wall, "job_s_extrapolated": job,
            "sample_fraction": {"spatial_frames": nframes / T, "temporal_modes": nmodes / Q}}


# ---------------------------------------------------------------------------
# accuracy check of the timed result (the metric's condition: <= 1e-6 vs FP64)
# ---------------------------------------------------------------------------
def sampled_columns(nkx: int) -> list:
    """kx columns whose modes (every ky) the accuracy check evaluates: DC, low q, and spread to Nyquist."""
    return sorted({0, 1, 2, 5, 17, nkx // 4, nkx // 2, nkx - 1} & set(range(nkx)))


def sampled_reference(frames: np.ndarray, lags, nx: int, ny: int, cols, window=None) -> np.ndarray:
    """D, PS, VAR at the kx columns `cols` (every ky, y-fftshifted) from direct FP64 DFTs of every frame.

    Rows of each frame against exp(-2 pi i x kx / nx), then columns against
    exp(-2 pi i y ky / ny), divided by sqrt(nx ny) (ddm.cc:319-323); D(lag) by
    direct differences (ddm.cc:118-146), PS = <|F|^2>_t and VAR from the
    mean-removed series, so the reference carries no Wiener-Khinchin
    cancellation.  Its own error is ~1e-16 sqrt(PS / D).
    """
    from concurrent.futures import ThreadPoolExecutor

    T, H, W = frames.shape
    C = len(cols)
    ex = np.exp(-2j * np.pi * np.outer(np.arange(W), np.asarray(cols)) / nx)
    exr = np.ascontiguousarray(np.concatenate([ex.real, ex.imag], axis=1))
    ey = np.exp(-2j * np.pi * np.outer(np.arange(ny), np.arange(H)) / ny)
    F = np.empty((T, ny, C), dtype=np.complex128)

    def rows(t0):
        blk = frames[t0:t0 + 16].astype(np.float64)
        if window is not None:
            blk *= window
        a = blk @ exr
        F[t0:t0 + 16] = np.einsum("yh,thc->tyc", ey, a[..., :C] + 1j * a[..., C:], optimize=True)

    threads = min(16, os.cpu_count() or 1)
    with ThreadPoolExecutor(max_workers=threads) as pool:
        list(pool.map(rows, range(0, T, 16)))
    F /= math.sqrt(float(nx * ny))
    Fq = F.reshape(T, ny * C)
    lags = [int(l) for l in lags]

    def modes(c0):
        f = Fq[:, c0:c0 + 256]
        o = np.empty((len(lags) + 2, f.shape[1]))
        for i, lag in enumerate(lags):
            d = f[lag:] - f[: T - lag]
            o[i] = (d.real * d.real + d.imag * d.imag).sum(axis=0) / float(T - lag)
        o[-2] = (f.real * f.real + f.imag * f.imag).sum(axis=0) / float(T)
        g = f - f.mean(axis=0)
        o[-1] = (g.real * g.real + g.imag * g.imag).sum(axis=0) / float(T)
        return o

    with ThreadPoolExecutor(max_workers=threads) as pool:
        parts = list(pool.map(modes, range(0, ny * C, 256)))
    return np.fft.fftshift(np.concatenate(parts, axis=1).reshape(len(lags) + 2, ny, C), axes=1)


def time_tier(DdmPlan, mode, T, H, W, code, lags, nx, ny, nt, window, precision, device, frames, stream, steps=2):
    """Device frames/s of one tier on the same stack (one warm-up step, CUDA events around `steps` steps)."""
    import torch

    plan = DdmPlan(mode, T, H, W, code, lags, nx, ny, nt if mode == "fft" else 0, window is not None, precision,
                   device)
    out = torch.empty(plan.out_shape, dtype=torch.float64, device=device)
    plan.run(frames, window, out, stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        plan.run(frames, window, out, stream)
    e1.record(stream)
    torch.cuda.synchronize(device)
    ms = e0.elapsed_time(e1) / steps
    del plan, out
    torch.cuda.empty_cache()
    return {"precision": precision, "value": T / (ms / 1000.0), "unit": "frames/s", "ms_per_step": ms,
            "steps": steps}


def half_plane(nx: int, ny: int):
    """|k| of the half plane, the pixels' counts in the full one, and the largest ky, as azimuthal_average sets
    them up."""
    kx = 2 * np.pi * np.fft.fftfreq(nx)[: nx // 2 + 1]
    ky = 2 * np.pi * np.fft.fftshift(np.fft.fftfreq(ny))
    counts = np.full((ny, nx // 2 + 1), 2)
    counts[:, 0] = 1
    counts[:, -1] = 1 if nx % 2 == 0 else 2
    gx, gy = np.meshgrid(kx, ky)
    return np.sqrt(gx ** 2 + gy ** 2), counts, ky[-1]


def azavg_record(out, nx: int, ny: int, device, bins: int = 512, reps: int = 3) -> dict:
    """The azimuthal average of the timed result (``bins`` bins over (0, ky[-1])), both kernel orders.

    Times the set-up as a call makes it (edges and weights on the host, bins, lists and
    per-bin sums on the device) and the average (one kernel, results left on the
    device), best of `reps`; reports the largest relative difference of the fast
    order against the bit-exact one.
    """
    import torch

    from fastddm_gb300 import azimuthalaverage as aa

    k, counts, k_max = half_plane(nx, ny)
    rec = {"bins": bins, "pixels": int(ny * (nx // 2 + 1)), "rows": int(out.shape[0]), "setup_ms": float("inf")}
    for _ in range(reps):
        torch.cuda.synchronize(device)
        t0 = time.perf_counter()
        args = aa.bin_arguments(k, bins, (0, k_max), None, None, counts, True)
        tables, _ = aa._bin_tables(k, args, True, device)
        torch.cuda.synchronize(device)
        rec["setup_ms"] = min(rec["setup_ms"], 1000 * (time.perf_counter() - t0))
    res = {}
    stream = torch.cuda.current_stream(device)
    for label, exact in (("exact", True), ("fast", False)):
        best = float("inf")
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            avg, err = aa._average(out, tables, args.n_bins, True, device, exact, False)
            e1.record(stream)
            torch.cuda.synchronize(device)
            best = min(best, e0.elapsed_time(e1))
        rec[f"{label}_ms"] = best
        res[label] = (avg, err)
    diff = 0.0
    for i in range(2):
        a, b = res["fast"][i], res["exact"][i]
        ok = ~torch.isnan(b)
        diff = max(diff, float(((a[ok] - b[ok]).abs() / b[ok].abs().clamp_min(1e-300)).max()))
    rec["fast_vs_exact_max_rel"] = diff
    return rec, device_azavg(out, nx, ny, device, bins)


def device_azavg(out, nx: int, ny: int, device, bins: int):
    """The azimuthal average of a structure function in device memory (``bins`` bins over
    (0, ky[-1]), the exact order), as an AzimuthalAverage with tau unset."""
    from fastddm_gb300 import azimuthalaverage as aa

    k, counts, k_max = half_plane(nx, ny)
    avg, err, mean, edges = aa.azimuthal_average_array(out, k, bins, (0, k_max), counts=counts, gpu_id=device.index or 0)
    return aa.AzimuthalAverage(avg, err, mean, None, edges)


def batch_fit_record(jobs, device, sample: int = 4) -> dict:
    """The fits of config 4's pipeline: each stack's azimuthal average (height / 4 bins) and one
    fit_multik_batch over all stacks (the reference's sweep for each, every sweep concurrent), against
    the oracle's sweeps on the first ``sample`` stacks (one host core; extrapolated to all stacks by
    their number of fits).  Set-up as in fit_record."""
    import torch

    from fastddm_gb300 import fit as gfit
    from fastddm_gb300 import fit_models

    sys.path.insert(0, str(ROOT / "oracle"))
    import fit_oracle as fo

    setups = []
    for j in jobs:
        av = device_azavg(j.out, j.nx, j.ny, device, max(8, j.shape[1] // 4))
        setups.append(fit_start(av, np.asarray(j.lags, dtype=np.float64), ref_frac=0.25))
    model = fit_models.simple_exponential_model
    bjobs = [dict(data=a, ref=ref, **kw) for a, ref, kw in setups]
    best, best_tot = float("inf"), float("inf")
    for _ in range(2):
        torch.cuda.synchronize(device)
        t0 = time.perf_counter()
        res = gfit.fit_multik_batch(bjobs, model)
        best_tot = min(best_tot, 1000 * (time.perf_counter() - t0))
        best = min(best, res[0][0].device_ms)
    nfits = [int(np.sum(~np.isnan(a.data[:, 0]))) + 1 for a, _, _ in setups]
    func, names, _ = fo.MODELS["simple_exponential_model"]
    t0 = time.perf_counter()
    par = []
    for (a, ref, kw), (tab, _) in list(zip(setups, res))[:sample]:
        params = fo.make_params("simple_exponential_model")
        for n in ("A", "B", "Gamma"):
            params[n]["value"] = float(kw[n])
        want = fo.fit_multik(func, names, params, a.tau, a.data, ref, err=a.err, use_err=True)
        par.append(fit_parity(tab, want, a, func))
    sample_ms = 1000 * (time.perf_counter() - t0)
    oracle_all = sample_ms * sum(nfits) / sum(nfits[:sample])
    return {"model": "simple_exponential_model", "stacks": len(jobs), "fits": int(sum(nfits)),
            "lags_range": [min(a.tau.size for a, _, _ in setups), max(a.tau.size for a, _, _ in setups)],
            "batch_device_ms": best, "batch_total_ms": best_tot,
            "success": int(sum(int(np.sum(t["success"])) for t, _ in res)),
            "oracle_sample_stacks": sample, "oracle_sample_ms": sample_ms,
            "oracle_all_ms_extrapolated": oracle_all, "oracle_cores": 1,
            "batch_vs_oracle": oracle_all / best,
            "parity_sample": {"k_well_determined": sum(p["k_well_determined"] for p in par),
                              "parity_max_over_tol": max(p["parity_max_over_tol"] for p in par),
                              "chi2_equal": sum(p["chi2_equal"] for p in par),
                              "chi2_device_lower": sum(p["chi2_device_lower"] for p in par),
                              "chi2_device_higher": sum(p["chi2_device_higher"] for p in par),
                              "success_agree": all(p["success_agree"] for p in par)}}


def fit_start(azavg, tau: np.ndarray, ref_frac: float = 0.125):
    """An azimuthal average set up for fit_multik as the reference's fit.py docstring does.

    Bins whose error is 0 or not finite (the k = 0 bin holds one pixel) become
    NaN rows; B from the "polyfit" noise estimate, A = 2 var - B and Gamma from
    the half-decay lag at the reference k.  Returns (data, ref, keyword arguments).
    """
    import copy as _copy

    from fastddm_gb300 import noise_est

    a = _copy.copy(azavg)
    a.tau = np.asarray(tau, dtype=np.float64)
    data = a._data.copy()
    bad = ~np.all(np.isfinite(a.err) & (a.err > 0), axis=1)
    data[bad, 0] = np.nan
    a._data = data
    B_est, _ = noise_est.estimate_camera_noise(a, mode="polyfit")
    valid = np.flatnonzero(~np.isnan(a.data[:, 0]))
    ref = int(valid[int(len(valid) * ref_frac)])
    A0 = 2.0 * a.var[ref] - B_est[ref]
    half = np.abs((a.data[ref] - B_est[ref]) / A0 - 0.5)
    G0 = 1.0 / a.tau[int(np.argmin(half))]
    return a, ref, dict(A=A0, B=B_est[ref], Gamma=G0, use_err=True)


def fit_parity(got, want, a, func) -> dict:
    """Device sweep against the oracle's: parameters on the k the oracle determines well (converged,
    A and Gamma to 10 %), over max(1e-5 of the scale, 0.1 standard error); chi^2 on every k, within
    max(1e-9 relative, 0.05 reduced chi^2)."""
    ok = ~np.isnan(want["A"])
    with np.errstate(invalid="ignore", divide="ignore"):
        rel = np.maximum(want["A_stderr"] / np.abs(want["A"]), want["Gamma_stderr"] / np.abs(want["Gamma"]))
    wd = ok & want["success"] & np.isfinite(rel) & (rel < 0.1)
    worst = 0.0
    for n in ("A", "B", "Gamma"):
        scale = np.abs(want["A"][wd]) if n == "B" else np.abs(want[n][wd])
        tol = np.maximum(1e-5 * scale, 0.1 * want[f"{n}_stderr"][wd])
        if wd.any():
            worst = max(worst, float(np.max(np.abs(got[n][wd] - want[n][wd]) / tol)))
    w = 1.0 / a.err
    with np.errstate(invalid="ignore", over="ignore"):
        chi_d = np.sum(((func(a.tau[None, :], got["A"][:, None], got["B"][:, None], got["Gamma"][:, None], 1.0)
                         - a.data) * w) ** 2, axis=1)
        chi_o = np.sum(((func(a.tau[None, :], want["A"][:, None], want["B"][:, None], want["Gamma"][:, None], 1.0)
                         - a.data) * w) ** 2, axis=1)
    ctol = np.maximum(1e-9 * chi_o, 0.05 * chi_o / (a.tau.size - 3))
    return {"k": int(ok.sum()), "k_well_determined": int(wd.sum()), "parity_max_over_tol": worst,
            "chi2_equal": int(np.sum(ok & (np.abs(chi_d - chi_o) <= ctol))),
            "chi2_device_lower": int(np.sum(ok & (chi_o - chi_d > ctol))),
            "chi2_device_higher": int(np.sum(ok & (chi_d - chi_o > ctol))),
            "success_agree": bool(np.array_equal(got["success"], want["success"]))}


def fit_record(azavg, tau: np.ndarray, reps: int = 3) -> dict:
    """fit_multik of the azimuthal average, as the reference's fit.py docstring sets it up.

    Simple exponential structure function, weights 1 / err, B from the
    "polyfit" noise estimate, A = 2 var - B and Gamma from the half-decay lag
    at the reference k.  Bins whose error is 0 or not finite (the k = 0 bin
    holds one pixel) are left out, as NaN rows.  Times the reference's
    sequential sweep (``warm_start="chain"``) and every k from the fit at ref
    (``"ref"``) on the device, best of ``reps``, and the oracle's sweep
    (lmfit's wrapper restated around scipy's MINPACK, one host core).  Parity:
    on the k the oracle determines well, the largest |device - oracle| over
    max(1e-5 of the scale, 0.1 standard error) (1 = at the tolerance); on every
    k, how many chi^2 agree within max(1e-9 relative, 0.05 reduced chi^2) and
    how many are lower or higher on the device.
    """
    from fastddm_gb300 import fit as gfit
    from fastddm_gb300 import fit_models

    sys.path.insert(0, str(ROOT / "oracle"))
    import fit_oracle as fo

    a, ref, kw = fit_start(azavg, tau)
    model = fit_models.simple_exponential_model
    rec = {"model": "simple_exponential_model", "lags": int(a.tau.size), "ref": ref, "use_err": True}
    tables = {}
    for order in ("chain", "ref"):
        best_dev, best_tot = float("inf"), float("inf")
        for _ in range(reps):
            t0 = time.perf_counter()
            tab, _ = gfit.fit_multik(a, model, ref, warm_start=order, **kw)
            best_tot = min(best_tot, 1000 * (time.perf_counter() - t0))
            best_dev = min(best_dev, tab.device_ms)
        rec[f"{order}_device_ms"] = best_dev
        rec[f"{order}_total_ms"] = best_tot
        rec[f"{order}_success"] = int(np.sum(tab["success"]))
        tables[order] = tab
    func, names, _ = fo.MODELS["simple_exponential_model"]
    params = fo.make_params("simple_exponential_model")
    for n in ("A", "B", "Gamma"):
        params[n]["value"] = float(kw[n])
    t0 = time.perf_counter()
    want = fo.fit_multik(func, names, params, a.tau, a.data, ref, err=a.err, use_err=True)
    rec["oracle_chain_ms"] = 1000 * (time.perf_counter() - t0)
    rec["oracle_cores"] = 1
    rec.update(fit_parity(tables["chain"], want, a, func))
    rec["chain_vs_oracle"] = rec["oracle_chain_ms"] / rec["chain_device_ms"]
    return rec


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------
class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}

        def num(x):
            try:
                return float(x)
            except ValueError:
                return None

        sm = [num(r[1]) for r in rows if num(r[1]) is not None]
        mx = [num(r[2]) for r in rows if num(r[2]) is not None]
        pw = [num(r[3]) for r in rows if num(r[3]) is not None]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "power_w_max": max(pw) if pw else None, "samples": len(rows), "reasons": reasons}


# ---------------------------------------------------------------------------
def side_record(f, *args):
    """A record beside the headline: an error in it is recorded, and the line still comes out."""
    try:
        return f(*args)
    except (ValueError, RuntimeError) as e:
        return {"error": f"{type(e).__name__}: {e}"}


def dist_setup():
    from fastddm_gb300 import replicas

    return replicas.world()


def run_reference(args):
    """CPU arm: the FP64 restatement of the reference's cpp core on every host core.

    Each step times a bounded sample of the workload (per worker: the spatial
    FFTs of 4 frames and the temporal stage of 2048 mode columns of the full
    length T) on all workers at once; `ms_per_step` is that sample's wall time
    and `value` the frames/s of the whole job extrapolated from the two
    measured rates.  The reference's own cpp core is not run: its FFT library
    (FFTW 3.3.10) builds only through CMake with a generated config.h, and its
    sources are not present where this benchmark runs.
    """
    _, rank, _ = module_alone("replicas").world()
    if rank != 0:
        return
    from concurrent.futures import ProcessPoolExecutor
    import multiprocessing as mp

    synthetic, next_fast_len = module_alone("synthetic"), module_alone("_fftopt").next_fast_len
    scene = getattr(synthetic, CONFIGS[args.config])
    lags = lags_for(args.config, scene.length)
    T, H, W = scene.length, scene.height, scene.width
    nx, ny, nt = next_fast_len(W, "cpp"), next_fast_len(H, "cpp"), next_fast_len(2 * T, "cpp")
    Q = ny * (nx // 2 + 1)
    small = synthetic.Scene(16, H, W, max(1, scene.n_spots), scene.sigma, scene.amplitude, scene.diffusivity,
                            scene.offset, scene.drift, scene.dtype, scene.seed)
    frames = synthetic.make_stack(small)
    workers = os.cpu_count() or 1
    samples = []
    with ProcessPoolExecutor(max_workers=workers, mp_context=mp.get_context("spawn")) as pool:
        for i in range(args.warmup + args.steps):
            r = cpu_throughput(frames, T, Q, nx, ny, nt, lags, workers, 4, 2048, pool)
            if i >= args.warmup:
                samples.append(r)
    value = statistics.mean(r["value"] for r in samples)
    sample_ms = 1000.0 * statistics.mean(r["sample_s"] for r in samples)
    frac = samples[0]["sample_fraction"]
    line = {
        "impl": "reference", "metric": "DDM frames/s", "value": value, "unit": "frames/s", "n_gpus": 0,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": sample_ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": workload_desc(args.config, scene, lags, "f64", "fft"),
        "cpu_baseline": {"value": value, "unit": "frames/s", "cores": workers, "kind": "port", "extrapolated": True,
                         "sample_fraction": frac, "sample_ms_per_step": sample_ms,
                         "job_ms_extrapolated": 1000.0 * T / value,
                         "sample": f"per step, on each of {workers} worker processes at once: the spatial FFTs of 4 "
                                   f"frames and the temporal stage of 2048 mode columns of {T} frames (numpy FP64 "
                                   f"restatement of the reference's cpp core, oracle/ddm_oracle.py); the job's time "
                                   f"is extrapolated as T / spatial rate + Q / temporal rate. The cpp core itself "
                                   f"is not built: FFTW builds only through CMake with a generated config.h"},
        "e2e": {"value": value, "unit": "frames/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def run_ours(args):
    import torch

    ws, rank, local = dist_setup()
    if ws > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    device = torch.device("cuda", local)
    torch.cuda.set_device(device)

    from fastddm_gb300 import _build, _lib, replicas, synthetic, window as fwin
    from fastddm_gb300._ddm_b200 import DdmPlan, ddm_diff_b200, ddm_fft_b200
    from fastddm_gb300._fftopt import next_fast_len

    _build.build()
    lib = _lib.load()
    scene = getattr(synthetic, CONFIGS[args.config])
    lags = lags_for(args.config, scene.length)
    T, H, W = scene.length, scene.height, scene.width
    nx, ny = next_fast_len(W, "b200"), next_fast_len(H, "b200")
    nt = next_fast_len(2 * T, "b200")
    nkx = nx // 2 + 1
    Q = ny * nkx
    L = len(lags)
    frames = synthetic.make_stack_torch(scene, device=device)
    code = {torch.uint8: 0, torch.int16: 1}.get(frames.dtype, 2)
    window = None
    if args.config == "medium":
        window = torch.from_numpy(fwin.blackman_harris((H, W))).to(device)
    plan = DdmPlan(args.mode, T, H, W, code, lags, nx, ny, nt if args.mode == "fft" else 0, window is not None,
                   args.precision, device)
    out = torch.empty(plan.out_shape, dtype=torch.float64, device=device)
    stream = torch.cuda.current_stream(device)
    for _ in range(args.warmup):
        plan.run(frames, window, out, stream)
    torch.cuda.synchronize(device)

    launches0 = lib.fddm_b200_launch_count()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(torch.cuda.current_device()) as clk:
        replicas.barrier()
        torch.cuda.synchronize(device)
        e0.record(stream)
        for _ in range(args.steps):
            plan.run(frames, window, out, stream)
        e1.record(stream)
        torch.cuda.synchronize(device)
        replicas.barrier()
    launches = int(lib.fddm_b200_launch_count() - launches0)
    ms = replicas.max_over_ranks(e0.elapsed_time(e1), device)
    ms_step = ms / args.steps
    value = replicas.aggregate_rate(T * args.steps, ms / 1000.0, ws)
    clocks = clk.summary()

    # the timed result's sampled modes, before any other run reuses the device
    cols = sampled_columns(nkx)
    got_cols = out[:, :, cols].cpu().numpy()

    # per-stage device times (untimed extra steps with CUDA events around each stage)
    import ctypes

    lib.fddm_b200_set_stage_timing(1)
    sp, tp = [], []
    for _ in range(2):
        plan.run(frames, window, out, stream)
        a, b = ctypes.c_float(), ctypes.c_float()
        _lib.check(lib.fddm_b200_stage_times(ctypes.byref(a), ctypes.byref(b)))
        sp.append(a.value)
        tp.append(b.value)
    lib.fddm_b200_set_stage_timing(0)
    sp_ms, tp_ms = statistics.mean(sp), statistics.mean(tp)

    # the plain all-FP64 GPU path on the same stack (the denominator of the >= 3x target) and diff
    # mode, whose result must agree with fft mode on every mode; both untimed against the metric
    f64 = None
    other = None
    if rank == 0 and not args.no_check:
        f64 = time_tier(DdmPlan, args.mode, T, H, W, code, lags, nx, ny, nt, window, "f64", device, frames, stream,
                        steps=2)
        if args.precision != "f64":
            f64["ff_speedup"] = value / ws / f64["value"]
        other_mode = "diff" if args.mode == "fft" else "fft"
        p2 = DdmPlan(other_mode, T, H, W, code, lags, nx, ny, nt if other_mode == "fft" else 0, window is not None,
                     args.precision, device)
        out2 = torch.empty(p2.out_shape, dtype=torch.float64, device=device)
        p2.run(frames, window, out2, stream)
        torch.cuda.synchronize(device)
        other = float(((out - out2).abs() / out2.abs()).max())
        del p2, out2
        torch.cuda.empty_cache()

    es = 16 if args.precision in ("ff", "f64") else 8
    b_in = frames.element_size()
    peaks = {}
    try:
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
        peak_src = "measured"
    except (OSError, ValueError):
        peak_src = "fallback"
    hbm = float(peaks.get("hbm_gbs", 6800.0))
    # algorithmic bytes per launch of the temporal kernel: read the spectrum once, write the output
    tfft_bytes = T * Q * es + (L + 2) * Q * 8
    # spatial stage (row + column passes): read frames, write the spectrum once
    spatial_bytes = T * H * W * b_in + T * Q * es
    job_bytes = T * H * W * b_in + 2 * T * Q * es + (L + 2) * Q * 8
    traffic = None
    tfile = ROOT / "profiles" / "traffic.json"
    if tfile.exists():
        try:
            traffic = json.loads(tfile.read_text()).get(f"{args.config}:{args.mode}:{args.precision}")
        except ValueError:
            traffic = None
    tkernel = "k_tdiff" if args.mode == "diff" else ("k_tfft_long" if args.config == "long" else "k_tfft")
    if args.precision == "ff":  # the float-float tier's kernels run in block fixed point
        tkernel = {"k_tdiff": "k_tdiff_fx", "k_tfft_long": "k_tfx_long", "k_tfft": "k_tfx"}[tkernel]
    dominant = tkernel if tp_ms >= sp_ms else "k_rows+k_cols"
    if dominant == tkernel:
        ach = tfft_bytes / (tp_ms / 1000.0) / 1e9
        tr = traffic.get(tkernel) if isinstance(traffic, dict) else None
    else:
        ach = spatial_bytes / (sp_ms / 1000.0) / 1e9
        tr = traffic.get("spatial") if isinstance(traffic, dict) else None
    roofline = {"bound": "hbm", "kernel": dominant, "achieved": ach, "peak": hbm, "unit": "GB/s",
                "frac": ach / hbm, "traffic": tr, "peak_source": peak_src,
                "stage_ms": {"spatial": sp_ms, "temporal": tp_ms},
                "job_bytes": job_bytes, "job_frac": job_bytes / (ms_step / 1000.0) / 1e9 / hbm}

    # instruction-issue roofline: the float-float FFTs are bound by the SM issue rate (4 warp
    # instructions per cycle per SM), not by HBM.  Warp instructions per mode / per frame come
    # from an ncu capture of the same kernel configuration; the times and the clock are live.
    issue = None
    ifile = ROOT / "profiles" / "instructions.json"
    if ifile.exists():
        try:
            ic = json.loads(ifile.read_text()).get(f"{args.config}:{args.mode}:{args.precision}")
        except ValueError:
            ic = None
        mhz = clocks.get("sm_mhz") if isinstance(clocks, dict) else None
        if ic and mhz:
            cyc = torch.cuda.get_device_properties(device).multi_processor_count * mhz * 1e6
            t_inst = ic["temporal_per_mode"] * Q
            s_inst = (ic["rows_per_frame"] + ic["cols_per_frame"]) * T
            t_rate = t_inst / (tp_ms / 1000.0) / cyc
            issue = {"bound": "sm_issue", "kernel": tkernel, "achieved": t_rate, "peak": 4.0,
                     "unit": "warp instructions/cycle/SM", "frac": t_rate / 4.0,
                     "spatial_frac": s_inst / (sp_ms / 1000.0) / cyc / 4.0,
                     "job_frac": (t_inst + s_inst) / (ms_step / 1000.0) / cyc / 4.0,
                     "sm_mhz": mhz, "source": ic["source"]}

    # the azimuthal average of the timed result (512 bins), both kernel orders
    azavg = fits = None
    if rank == 0 and not args.no_check:
        rec = side_record(azavg_record, out, nx, ny, device)
        azavg, aa_obj = rec if isinstance(rec, tuple) else (rec, None)
        if aa_obj is not None:
            fits = side_record(fit_record, aa_obj, np.asarray(lags, dtype=np.float64))

    # end to end through the public API: pinned host frames in, host result out
    e2e = None
    if not args.no_e2e and rank == 0:
        host = torch.empty(frames.shape, dtype=frames.dtype, pin_memory=True)
        host.copy_(frames)
        del plan, out
        torch.cuda.empty_cache()
        wnp = window.cpu().numpy() if window is not None else np.array([], dtype=np.float64)
        if args.mode == "fft":
            def fn(x):
                return ddm_fft_b200(x, lags, nx, ny, nt, wnp, precision=args.precision)
        else:
            def fn(x):
                return ddm_diff_b200(x, lags, nx, ny, wnp, precision=args.precision)
        for _ in range(max(2, args.warmup)):  # warm-up: device and page-locked allocator caches
            res = fn(host)
            del res
        times = []
        for _ in range(max(1, args.steps)):
            torch.cuda.synchronize(device)
            t0 = time.perf_counter()
            res = fn(host)
            times.append(time.perf_counter() - t0)
            nbytes_out = res.nbytes
            del res
        e2e = {"value": T / statistics.mean(times), "unit": "frames/s",
               "h2d_bytes_per_step": int(host.numel() * host.element_size()),
               "d2h_bytes_per_step": int(nbytes_out), "ms_per_step": 1000 * statistics.mean(times),
               "step_ms": [round(1000 * t, 2) for t in times]}

    # end to end from a plain (pageable) numpy stack: the call a FastDDM user makes with an array in
    # hand; the frames go through the copy-engine upload, overlapped with the spatial stage
    e2e_pageable = None
    if not args.no_e2e and rank == 0:
        hnp = frames.cpu().numpy() if frames.dtype == torch.uint8 else frames.to(torch.int32).cpu().numpy().astype(
            np.uint16)
        times = []
        for i in range(max(1, args.steps) + 1):
            torch.cuda.synchronize(device)
            t0 = time.perf_counter()
            res = fn(hnp)
            if i > 0:  # the first call warms the page-locked result buffer
                times.append(time.perf_counter() - t0)
            del res
        e2e_pageable = {"value": T / statistics.mean(times), "unit": "frames/s",
                        "h2d_bytes_per_step": int(hnp.nbytes), "d2h_bytes_per_step": int(nbytes_out),
                        "ms_per_step": 1000 * statistics.mean(times), "step_ms": [round(1000 * t, 2) for t in times],
                        "input": "pageable numpy array (copy-engine upload overlapped with the row pass)"}

    # accuracy of the timed result against direct FP64 DFTs of every frame at the sampled modes
    accuracy = None
    if rank == 0 and not args.no_check:
        host_frames = frames.cpu().numpy() if frames.dtype == torch.uint8 else frames.to(torch.int32).cpu().numpy()
        wref = window.cpu().numpy() if window is not None else None
        exact = sampled_reference(host_frames, lags, nx, ny, cols, wref)
        del host_frames
        err = np.abs(got_cols - exact) / np.abs(exact)
        nodc = err.copy()
        nodc[:, ny // 2, cols.index(0)] = 0.0
        worst = max(float(err.max()), other if other is not None else 0.0)
        accuracy = {"max_rel_err": worst, "target": 1e-6, "ok": worst <= 1e-6,
                    f"{args.mode}_vs_fp64_dft": float(err.max()), f"{args.mode}_vs_fp64_dft_noDC": float(nodc.max()),
                    "sampled_modes": int(ny * len(cols)), "kx_columns": cols,
                    f"{args.mode}_vs_{'diff' if args.mode == 'fft' else 'fft'}_all_modes": other,
                    "reference": "direct FP64 DFTs of every timed frame at the sampled kx columns (all ky), D by "
                                 "direct differences, PS and VAR from the mean-removed series (ddm.cc:118-164)"}

    cpu = None
    if not args.no_cpu and rank == 0 and ws == 1:
        sample = frames[:32].cpu().numpy()
        r = cpu_throughput(sample, T, Q, nx, ny, nt, lags, 1, 32, 16384, None)
        cpu = {"value": r["value"], "unit": "frames/s", "cores": 1, "kind": "port", "extrapolated": True,
               "sample_fraction": r["sample_fraction"], "sample_s": r["sample_s"],
               "sample": f"spatial FFT of 32 frames and the temporal stage of 16384 mode columns x {T} frames "
                         f"(FP64 numpy restatement of the cpp core), extrapolated to the full job"}

    serve = None
    if rank == 0 and ws == 1 and not args.no_serve and args.config == "large":
        del frames
        torch.cuda.empty_cache()
        serve = side_record(serve_records, args, args.requests, device)

    if rank == 0:
        line = {
            "metric": "DDM frames/s", "value": value, "unit": "frames/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": {"ff": "ff (float-float)", "f64": "f64", "f32": "f32"}[args.precision],
            "data": "synthetic", "config": workload_desc(args.config, scene, lags, args.precision, args.mode),
            "roofline": roofline, "issue_roofline": issue, "cpu_baseline": cpu, "e2e": e2e,
            "e2e_pageable": e2e_pageable, "accuracy": accuracy,
            "max_rel_err": accuracy["max_rel_err"] if accuracy else None, "f64_path": f64, "serve": serve,
            "azimuthal_average": azavg, "fit_multik": fits,
            "clocks": clocks, "gpu_launches": launches,
        }
        print(json.dumps(line))
        if accuracy is not None and not accuracy["ok"]:
            sys.exit(f"max relative error {accuracy['max_rel_err']:.3e} exceeds the metric's 1e-6")
    if ws > 1:
        torch.distributed.destroy_process_group()


def run_validate(args):
    """Max relative error of the b200 result on a sample of Fourier modes of the full workload.

    The reference values come from direct FP64 DFTs of every frame at the
    sampled modes (8 kx columns including kx = 0, all ky) and the direct
    difference formula for D (no Wiener-Khinchin cancellation), PS and VAR.
    """
    import torch

    sys.path.insert(0, str(ROOT / "oracle"))
    import ddm_oracle as oracle
    from fastddm_gb300 import synthetic, window as fwin
    from fastddm_gb300._ddm_b200 import DdmPlan
    from fastddm_gb300._fftopt import next_fast_len

    device = torch.device("cuda", 0)
    scene = getattr(synthetic, CONFIGS[args.config])
    lags = lags_for(args.config, scene.length)
    T, H, W = scene.length, scene.height, scene.width
    nx, ny, nt = next_fast_len(W, "b200"), next_fast_len(H, "b200"), next_fast_len(2 * T, "b200")
    nkx = nx // 2 + 1
    frames = synthetic.make_stack_torch(scene, device=device)
    code = {torch.uint8: 0, torch.int16: 1}.get(frames.dtype, 2)
    wnp = fwin.blackman_harris((H, W)) if args.config == "medium" else None
    window = torch.from_numpy(wnp).to(device) if wnp is not None else None
    results = {}
    outs = {}
    for mode, prec in (("fft", args.precision), ("diff", args.precision), ("fft", "f64"), ("fft", "f32")):
        plan = DdmPlan(mode, T, H, W, code, lags, nx, ny, nt if mode == "fft" else 0, window is not None, prec, device)
        out = torch.empty(plan.out_shape, dtype=torch.float64, device=device)
        plan.run(frames, window, out)
        torch.cuda.synchronize()
        outs[(mode, prec)] = out.cpu().numpy()
        del plan, out
        torch.cuda.empty_cache()
    # sampled exact spectra: columns kx in `cols`, every ky
    cols = sorted({0, 1, 2, 5, 17, nkx // 4, nkx // 2, nkx - 1})
    ex = np.exp(-2j * np.pi * np.outer(np.arange(W), np.array(cols)) / nx)          # (W, C)
    ey = np.exp(-2j * np.pi * np.outer(np.fft.fftfreq(ny) * ny, np.arange(H)) / ny)  # (ny, H)
    Fs = np.empty((T, ny, len(cols)), dtype=np.complex128)
    host = frames.cpu().numpy()
    for t0 in range(0, T, 64):
        blk = host[t0:t0 + 64].astype(np.float64)
        if wnp is not None:
            blk = blk * wnp
        Fs[t0:t0 + 64] = (ey @ (blk @ ex)) / math.sqrt(nx * ny)
    Fq = Fs.reshape(T, -1)
    exact = oracle.temporal_diff(Fq, lags)  # D by differences; VAR recomputed below without cancellation
    G = Fq - Fq.mean(axis=0)
    exact[-1] = (G.real ** 2 + G.imag ** 2).mean(axis=0)
    exact = exact.reshape(len(lags) + 2, ny, len(cols))
    exact = np.fft.fftshift(exact, axes=1)
    for key, out in outs.items():
        got = out[:, :, cols]
        e = np.abs(got - exact) / np.abs(exact)
        e_nodc = e.copy()
        e_nodc[:, ny // 2, cols.index(0)] = 0
        results[f"{key[0]}_{key[1]}"] = {"max_rel": float(e.max()), "max_rel_noDC": float(e_nodc.max()),
                                         "median_rel": float(np.median(e))}
    a, b = outs[("fft", args.precision)], outs[("diff", args.precision)]
    results["fft_vs_diff_all_modes"] = float(np.max(np.abs(a - b) / np.abs(b)))
    results["fft_vs_f64_all_modes"] = float(np.max(np.abs(a - outs[("fft", "f64")]) / np.abs(outs[("fft", "f64")])))
    print(json.dumps({"validate": args.config, "sampled_modes": len(cols) * ny, "kx_columns": cols,
                      "lags": int(len(lags)), "errors": results}))


def _clock_block(clk):
    return clk.summary() if clk is not None else None


def run_batch(args):
    """96 uneven stacks (sides 64..512, 100..2000 frames, uint16, all lags) in one batch call."""
    import torch

    from fastddm_gb300 import _build, _lib, synthetic, batch as fb
    from fastddm_gb300._ddm_b200 import DdmPlan

    _build.build()
    lib = _lib.load()
    device = torch.device("cuda", 0)
    scenes = synthetic.config4_scenes(96, seed=0)
    jobs = []
    for sc in scenes:
        frames = synthetic.make_stack_torch(sc, device=device)
        jobs.append(fb.make_job(frames, np.arange(1, sc.length), mode=args.mode, device=device))
    total_frames = sum(sc.length for sc in scenes)
    stream = torch.cuda.current_stream(device)
    # kernels of one batch launch (the graph replays the same launches)
    plan = fb.BatchPlan(jobs, args.precision, device, graph=True)
    l0 = lib.fddm_b200_launch_count()
    plan._launch(stream)
    per_batch = int(lib.fddm_b200_launch_count() - l0)
    for _ in range(max(1, args.warmup)):  # the first run captures the CUDA graph
        plan.run(stream)
    torch.cuda.synchronize(device)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(0) as clk:
        e0.record(stream)
        for _ in range(args.steps):
            plan.run(stream)
        e1.record(stream)
        torch.cuda.synchronize(device)
    ms = e0.elapsed_time(e1) / args.steps
    launches = per_batch * args.steps
    value = total_frames / (ms / 1000.0)
    batch_out = [j.out.clone() for j in jobs]
    # the same jobs one at a time on one stream: plans built before the timed region, no host sync between jobs
    del plan
    torch.cuda.empty_cache()
    plans = [DdmPlan(j.mode, *j.shape, j.dtype_code, j.lags, j.nx, j.ny, j.nt, False, args.precision, device)
             for j in jobs]
    for j, p in zip(jobs, plans):
        p.run(j.frames, None, j.out, stream)
    torch.cuda.synchronize(device)
    seq = []
    for _ in range(max(1, min(args.steps, 3))):
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        for j, p in zip(jobs, plans):
            p.run(j.frames, None, j.out, stream)
        t1.record(stream)
        torch.cuda.synchronize(device)
        seq.append(t0.elapsed_time(t1))
    seq_ms = min(seq)
    identical = all(bool(torch.equal(a, j.out)) for a, j in zip(batch_out, jobs))
    del plans, batch_out
    fits = side_record(batch_fit_record, jobs, device)
    line = {
        "metric": "DDM frames/s (batched uneven stacks)", "value": value, "unit": "frames/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": args.precision, "data": "synthetic",
        "config": {"workload": f"batch_{len(scenes)}_stacks_{total_frames}_frames_all_lags", "stacks": len(scenes),
                   "frames": total_frames, "mode": args.mode, "precision": args.precision,
                   "sides": sorted({sc.height for sc in scenes}), "frames_range": [min(s.length for s in scenes),
                                                                                   max(s.length for s in scenes)]},
        "one_at_a_time": {"value": total_frames / (seq_ms / 1000.0), "ms": seq_ms,
                          "how": "the same jobs through per-stack plans built before timing, back to back on one "
                                 "stream without host syncs (best of up to 3 passes)"},
        "batch_over_one_at_a_time": seq_ms / ms, "results_identical_to_one_at_a_time": identical,
        "graph": "CUDA graph of fddm_b200_batch_launch, replayed each step", "fit_multik_batch": fits,
        "clocks": _clock_block(clk), "gpu_launches": launches,
    }
    print(json.dumps(line))


def serve_records(args, n_req: int, device) -> dict:
    """Poisson arrivals (50 req/s) of config-4-sized jobs plus 5 % 1024^2 x 2000 jobs, served twice:
    continuous batching in the float-float tier, and one request at a time in the FP64 tier."""
    import torch

    from fastddm_gb300 import synthetic
    from fastddm_gb300._ddm_b200 import DdmPlan
    from fastddm_gb300.serving import DdmServer, GpuExecutor, Request, latency_summary, replay

    rng = np.random.default_rng(7)
    scenes = synthetic.config4_scenes(n_req, seed=100)
    big = rng.random(n_req) < 0.05
    scenes = [synthetic.Scene(2000, 1024, 1024, 1024 * 1024 // 82, 2.0, 2000.0, 0.5, 500.0, 0.0, "uint16", 900 + i)
              if big[i] else sc for i, sc in enumerate(scenes)]
    arrivals = np.cumsum(rng.exponential(1.0 / 50.0, n_req))
    frames = [synthetic.make_stack_torch(sc, device=device) for sc in scenes]
    torch.cuda.synchronize(device)
    total_frames = sum(sc.length for sc in scenes)
    checked = list(range(0, n_req, max(1, n_req // 8)))[:8]

    def requests(scale):
        return [Request(i, frames[i], np.arange(1, scenes[i].length), "fft", None, float(arrivals[i] * scale))
                for i in range(n_req)]

    results = {}
    # the stream as specified; the same stream arriving 10x faster (a queue forms, so small requests
    # admitted together share a batched launch); one request at a time in FP64
    for label, prec, streams, scale in (("continuous_batching", args.precision, 6, 1.0),
                                        ("continuous_batching_10x_rate", args.precision, 6, 0.1),
                                        ("one_at_a_time_f64", "f64", 1, 1.0)):
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info(device)
        ex = GpuExecutor(0, prec, streams, pool_bytes=int(0.35 * free))
        server = DdmServer(ex, int(0.85 * free), small_bytes=512 << 20) if streams > 1 else \
            DdmServer(ex, int(0.85 * free), small_bytes=0)
        # warm-up: FFT tables of every frame size and every temporal length in the stream
        for side in sorted({sc.height for sc in scenes}):
            p = DdmPlan("fft", 8, side, side, 2, np.arange(1, 8), side, side, 16, False, prec, device)
            f = torch.zeros((8, side, side), dtype=frames[0].dtype, device=device)
            p.run(f, None, torch.empty(p.out_shape, dtype=torch.float64, device=device))
        for T in sorted({sc.length for sc in scenes}):
            p = DdmPlan("fft", T, 2, 2, 2, np.arange(1, T), 2, 2, 2 * T, False, prec, device)
            f = torch.zeros((T, 2, 2), dtype=frames[0].dtype, device=device)
            p.run(f, None, torch.empty(p.out_shape, dtype=torch.float64, device=device))
        torch.cuda.synchronize(device)
        ex.clock_start()
        kept = {}

        def deliver(r):  # the client takes each result; a few are kept for the identity check
            res = server.fetch(r.rid)
            if r.rid in checked and label.startswith("continuous_batching"):
                kept[r.rid] = res

        reqs = replay(server, requests(scale), time.perf_counter, deliver=deliver)
        span = max(r.completed for r in reqs) - min(r.arrival for r in reqs)
        summ = latency_summary(reqs)
        summ.update({"frames_per_s": total_frames / span, "span_s": span, "peak_inflight": server.peak_inflight,
                     "batched_launches": server.batches, "slots": streams, "precision": prec,
                     "arrival_rate_per_s": 50.0 / scale})
        results[label] = summ
        if label.startswith("continuous_batching"):
            # a few results again, each alone on an idle device: must be identical
            same = True
            for i in checked:
                sc = scenes[i]
                p = DdmPlan("fft", sc.length, sc.height, sc.width, 2, np.arange(1, sc.length), sc.width, sc.height,
                            2 * sc.length, False, prec, device)
                alone = torch.empty(p.out_shape, dtype=torch.float64, device=device)
                p.run(frames[i], None, alone)
                torch.cuda.synchronize(device)
                same = same and bool(torch.equal(alone, kept[i]))
                del p, alone
            results[label]["identical_alone_and_in_mix"] = same
        del server, ex, reqs, kept
    del frames
    torch.cuda.empty_cache()
    cb, one = results["continuous_batching"], results["one_at_a_time_f64"]
    return {"requests": n_req, "arrivals": "Poisson, mean 50 requests/s", "large_jobs": int(big.sum()),
            "frames": total_frames, "mode": "fft", "all_lags": True,
            "p50_ms": cb["p50_ms"], "p99_ms": cb["p99_ms"], "frames_per_s": cb["frames_per_s"],
            "vs_one_at_a_time_f64_frames_per_s": cb["frames_per_s"] / one["frames_per_s"], "legs": results}


def run_serve(args):
    import torch

    from fastddm_gb300 import _build

    _build.build()
    rec = serve_records(args, args.requests, torch.device("cuda", 0))
    line = {
        "metric": "serve p50/p99 latency", "value": rec["p99_ms"], "unit": "ms (p99)", "n_gpus": 1,
        "higher_is_better": False, "dtype": args.precision, "data": "synthetic",
        "config": {"workload": f"serve_{args.requests}_requests_poisson_50_per_s", "requests": args.requests,
                   "large_jobs": rec["large_jobs"], "frames": rec["frames"], "mode": "fft"},
        "serve": rec,
    }
    print(json.dumps(line))


def run_dft_stage(args):
    """The first radix-32 stage of the row transform of 1024-pixel 8-bit rows, two ways: the two
    float-float butterfly passes, and the CUDA-core work a 5-slice bf16 DFT-as-GEMM stage would still
    need (slice-sum combination, row packing, twiddle; no MMA: a lower bound on its time)."""
    import torch

    from fastddm_gb300 import _build, _lib

    _build.build()
    lib = _lib.load()
    device = torch.device("cuda", 0)
    npairs = 32768  # 64 frames of 1024 x 1024
    g = torch.Generator(device=device)
    g.manual_seed(0)
    rows = torch.randint(0, 256, (npairs * 2 * 1024,), dtype=torch.uint8, device=device, generator=g)
    out = torch.empty((npairs * 1024 * 16,), dtype=torch.uint8, device=device)
    stream = torch.cuda.current_stream(device)
    res = {}
    for variant, label in ((0, "float_float_butterflies"), (1, "tensor_stage_cuda_core_floor")):
        for _ in range(args.warmup):
            _lib.check(lib.fddm_b200_experiment_dft_stage(variant, rows.data_ptr(), npairs, out.data_ptr(),
                                                          stream.cuda_stream))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            _lib.check(lib.fddm_b200_experiment_dft_stage(variant, rows.data_ptr(), npairs, out.data_ptr(),
                                                          stream.cuda_stream))
        e1.record(stream)
        torch.cuda.synchronize(device)
        ms = e0.elapsed_time(e1) / args.steps
        res[label] = {"ms_per_launch": ms, "us_per_frame": 1000 * ms / 64}
    res["floor_over_butterflies"] = res["tensor_stage_cuda_core_floor"]["ms_per_launch"] / \
        res["float_float_butterflies"]["ms_per_launch"]
    print(json.dumps({"measurement": "dft_stage", "rows": npairs * 2, "row_length": 1024, "frames": 64,
                      "steps": args.steps, "results": res}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="large", choices=sorted(CONFIGS))
    ap.add_argument("--mode", default="fft", choices=["fft", "diff"])
    ap.add_argument("--precision", default="ff", choices=["ff", "f64", "f32"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-check", action="store_true", help="skip the accuracy check and the f64/other-mode runs")
    ap.add_argument("--no-serve", action="store_true", help="skip the serving record of the default line")
    ap.add_argument("--validate", action="store_true", help="report sampled errors against exact FP64 spectra")
    ap.add_argument("--requests", type=int, default=100, help="serve: number of requests")
    args = ap.parse_args()
    if args.validate:
        run_validate(args)
    elif args.config == "batch":
        run_batch(args)
    elif args.config == "serve":
        run_serve(args)
    elif args.config == "dft_stage":
        run_dft_stage(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
