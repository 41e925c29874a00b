#!/usr/bin/env python
"""RoadRunner transit-model throughput on GB300.

Workload (one "step" = one evaluation of the model for a whole population):
8192 parameter vectors x 19,700 times (2-min cadence over 27.4 d at BJD
2459000), four contiguous light curves in four passbands, quadratic limb
darkening, nsamples = 1; k ~ U(0.05, 0.15), t0 ~ 2459000 + N(0, 1e-3),
p ~ U(0.5, 15), a ~ U(3, 20), b ~ U(0, 0.9), e = w = 0; seeded synthetic data.

Reported (one JSON line from rank 0):
  value      model points/s of the split-precision path, inputs resident in HBM
             (LD tables + prologue + flux kernels per step, CUDA events);
  e2e        the same through the public API (RoadRunnerModel.evaluate) with
             host parameter arrays in and the flux copied to pinned host memory;
  fp64       the plain all-FP64 GPU path on the same inputs;
  roofline   the flux kernel's algorithmic bytes / its event-timed duration
             against the measured HBM copy bandwidth;
  cpu_baseline  the oracle's FP64 C port (OpenMP, all host cores) on a
             bounded sample of the same workload, and at 1 thread (the
             reference's default nthreads=1) on a smaller sample;
  parity_vs_oracle  the GPU's FP64 and split results for the whole workload
             against the oracle's FP64 flux of the same workload;
  serve      the serving leg: a Poisson stream of the mixed-request workload
             through RRServer (p50/p99 latency, offered vs achieved rate, the
             highest sustained rate, vs the plain FP64 path per request);
  c2_precision / c3_gradient / ts / eclipse  the other workloads.
``--impl reference`` times that CPU implementation alone (the reference's
path restated in C; the reference itself is Python + numba, absent here).
"""
import argparse
import gc
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

WORKLOAD = ("8192 parameter vectors x 19700 times (2-min cadence, 27.4 d, BJD 2459000), "
            "4 light curves / passbands, quadratic LD, nsamples=1")
METRIC = "model points/s (RoadRunner flux values per second)"


def workload(npv=8192, npt=19700, seed=1234):
    rng = np.random.default_rng(seed)
    T = 2459000.0
    nlc = 4
    time_ = T + np.arange(npt) * (2.0 / 1440.0)
    lcids = np.minimum((np.arange(npt) * nlc) // npt, nlc - 1).astype(np.int64)
    k = rng.uniform(0.05, 0.15, (npv, 1))
    ldc = np.stack([rng.uniform(0, .6, (npv, nlc)), rng.uniform(0, .3, (npv, nlc))], -1)
    t0 = T + rng.normal(0, 1e-3, (npv, 1))
    p = rng.uniform(0.5, 15.0, npv)
    a = rng.uniform(3.0, 20.0, npv)
    inc = np.arccos(rng.uniform(0.0, 0.9, npv) / a)
    e = np.zeros(npv)
    w = np.zeros(npv)
    data = dict(time=time_, lcids=lcids, pbids=np.arange(nlc), nsamples=np.ones(nlc, int),
                exptimes=np.zeros(nlc))
    return data, dict(k=k, ldc=ldc, t0=t0, p=p, a=a, i=inc, e=e, w=w)


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def profiled_traffic(npv, npt):
    """DRAM bytes per launch of the split flux kernel from the committed ncu
    summary of that kernel (its traffic_bytes_per_point line), scaled to this
    launch's points."""
    path = os.path.join(ROOT, "profiles", "flux_split_c1.md")
    if not os.path.exists(path):
        return None
    vals = {}
    with open(path) as f:
        for line in f:
            if line.startswith("traffic_bytes_per_point:"):
                vals["bpp"] = float(line.split(":")[1])
    if "bpp" not in vals:
        return None
    return vals["bpp"] * npv * npt


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
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
        if self.proc is None or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        rows = []
        with open(self.path) as f:
            for line in f:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 8:
                    rows.append(parts)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        smax = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[j] for r in rows for j in range(4) if r[4 + j].lower() == "active"})
        pw = [float(r[3]) for r in rows if r[3].replace(".", "").isdigit()]
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": reasons, "samples": len(rows), "sm_mhz_min": min(sm) if sm else None,
                "power_w_max": max(pw) if pw else None}


def cpu_rr_full(model, prm, npv_sample, nthreads):
    import oracle
    ldp, istar = oracle.evaluate_ld_named('quadratic', model.mu, prm["ldc"][:npv_sample])
    sl = slice(0, npv_sample)
    return oracle.rr_full(model.time, prm["k"][sl], prm["t0"][sl], prm["p"][sl], prm["a"][sl], prm["i"][sl],
                          prm["e"][sl], prm["w"][sl], model.nlc, model.npb, model.nep, model.lcids,
                          model.pbids, model.epids, model.nsamples, model.exptimes, ldp, istar,
                          model.weights, model.dk, model.klims[0], model.klims[1], model.dg, model.ze,
                          nthreads=nthreads)


def cpu_oracle_model(data):
    import oracle
    m = oracle.OracleRoadRunner('quadratic')
    m.set_data(**data)
    return m


def run_cpu_baseline(data, prm, budget_s=12.0, npv_sample=8192, keep=None):
    """The oracle's C port of rr_full on all host cores, on the first
    npv_sample parameter vectors of the workload, repeated for ~budget_s.
    keep: a dict that receives the flux of the first repetition (the FP64
    result the GPU paths are checked against)."""
    ncores = os.cpu_count() or 1
    m = cpu_oracle_model(data)
    cpu_rr_full(m, prm, 16, ncores)          # warm-up (thread pool, pages)
    reps, t_total = 0, 0.0
    while t_total < budget_s and reps < 1000:
        t = time.perf_counter()
        f = cpu_rr_full(m, prm, npv_sample, ncores)
        t_total += time.perf_counter() - t
        if reps == 0 and keep is not None:
            keep["flux"] = f
        del f
        reps += 1
    npt = data["time"].size
    value = reps * npv_sample * npt / t_total
    # the reference's default is one thread (nthreads=1): a bounded sample at 1 thread beside it
    npv_1, reps_1, t_1 = 256, 0, 0.0
    while t_1 < 3.0 and reps_1 < 100:
        t = time.perf_counter()
        cpu_rr_full(m, prm, npv_1, 1)
        t_1 += time.perf_counter() - t
        reps_1 += 1
    value_1 = reps_1 * npv_1 * npt / t_1
    return {"value": value, "unit": "model points/s", "cores": ncores, "kind": "port",
            "sample": f"{npv_sample} of 8192 parameter vectors x {npt} times, {reps} repetitions, "
                      f"{t_total:.1f} s (oracle/rr_oracle.c rr_full restatement, OpenMP, FP64)",
            "value_1_thread": value_1,
            "sample_1_thread": f"{npv_1} parameter vectors x {npt} times, {reps_1} repetitions, {t_1:.1f} s"}


def impl_reference(args, rank):
    if rank != 0:
        return 0
    data, prm = workload()
    ncores = os.cpu_count() or 1
    m = cpu_oracle_model(data)
    npv_sample = prm["p"].size             # the whole population: the same workload as the GPU arm
    npt = data["time"].size
    for _ in range(args.warmup):
        cpu_rr_full(m, prm, npv_sample, ncores)
    t = time.perf_counter()
    for _ in range(args.steps):
        cpu_rr_full(m, prm, npv_sample, ncores)
    dt = time.perf_counter() - t
    value = args.steps * npv_sample * npt / dt
    sample = (f"all {npv_sample} parameter vectors x {npt} times per step (oracle/rr_oracle.c "
              f"rr_full restatement, OpenMP on {ncores} host threads, FP64)")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "model points/s",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * dt / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": WORKLOAD, "npv_per_gpu": npv_sample, "npt": npt, "npb": 4, "nlc": 4,
                       "nsamples": 1, "ld": "quadratic", "precision": "fp64"},
            "cpu_baseline": {"value": value, "unit": "model points/s", "cores": ncores, "kind": "port",
                             "sample": sample},
            "e2e": {"value": value, "unit": "model points/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# Other workloads: precision form (C2), differentiation (C3), serving (C4)
# ---------------------------------------------------------------------------

def c2_workload(npv=4096, seed=2024):
    """16 light curves, npt log-uniform in [500, 50000] at 30-min cadence from BJD
    2459000, nsamples = 10 with 30-min exposures, passbands j mod 4; power-2 LD;
    eccentric orbits; other parameters as the default workload."""
    rng = np.random.default_rng(seed)
    T = 2459000.0
    npts = np.exp(rng.uniform(np.log(500), np.log(50000), 16)).astype(int)
    time_ = np.concatenate([T + np.arange(n) / 48.0 for n in npts])
    lcids = np.concatenate([np.full(n, j) for j, n in enumerate(npts)])
    data = dict(time=time_, lcids=lcids, pbids=np.arange(16) % 4, nsamples=np.full(16, 10),
                exptimes=np.full(16, 1 / 48))
    a = rng.uniform(3.0, 20.0, npv)
    prm = dict(k=rng.uniform(0.05, 0.15, (npv, 1)),
               ldc=np.stack([rng.uniform(.3, .9, (npv, 4)), rng.uniform(.3, .8, (npv, 4))], -1),
               t0=T + rng.normal(0, 1e-3, (npv, 1)), p=rng.uniform(0.5, 15.0, npv), a=a,
               i=np.arccos(rng.uniform(0.0, 0.9, npv) / a), e=rng.uniform(0, 0.3, npv),
               w=rng.uniform(0, 2 * np.pi, npv))
    return data, prm


def bench_model(model, prm, steps, torch, device):
    """Mean ms of model.evaluate(copy=False) (parameters uploaded each call)."""
    args = (prm["k"], prm["ldc"], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"], prm["w"])
    out = model.evaluate(*args, copy=False)
    torch.cuda.synchronize(device)
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    t0.record()
    for _ in range(steps):
        out = model.evaluate(*args, copy=False)
    t1.record()
    torch.cuda.synchronize(device)
    return t0.elapsed_time(t1) / steps, out


def bench_c2(torch, device, steps=5, n_oracle=256):
    from pytransit_gb300 import RoadRunnerModel
    data, prm = c2_workload()
    npv, npt = prm["p"].size, data["time"].size
    res = {}
    for prec in ("split", "fp64"):
        m = RoadRunnerModel('power-2', precision=prec, device=device)
        m.fp64_cull = False      # the plain FP64 path is the comparator
        m.set_data(**data)
        ms, out = bench_model(m, prm, steps if prec == "split" else 2, torch, device)
        res[prec] = (ms, out)
        if prec == "fp64":
            # the drop-in's precision='fp64': the same arithmetic, the fold once per tile
            m.fp64_cull = True
            ms_c, out_c = bench_model(m, prm, 2, torch, device)
            culled_same = bool(torch.equal(out_c.nan_to_num(7.0), out.nan_to_num(7.0)))
            res["fp64_culled"] = (ms_c, None)
            del out_c
    dF = float((res["split"][1].double() - res["fp64"][1]).abs().max().item())
    # a seeded subset of the population against the oracle (the reference's
    # algorithm in FP64 C on the host cores), on the full C2 data
    import oracle
    sub = np.sort(np.random.default_rng(7).choice(npv, n_oracle, replace=False))
    ref = oracle.OracleRoadRunner('power-2')
    ref.set_data(**data)
    t = time.perf_counter()
    want = ref.evaluate(*(prm[n][sub] for n in ("k", "ldc", "t0", "p", "a", "i", "e", "w")))
    t_oracle = time.perf_counter() - t
    sub_t = torch.as_tensor(sub, device=device)
    got64 = res["fp64"][1].index_select(0, sub_t).cpu().numpy()
    got32 = res["split"][1].index_select(0, sub_t).double().cpu().numpy()
    pts = npv * npt
    return {"workload": f"{npv} pv x {npt} times (16 light curves, 30-min cadence, 10 supersamples, 4 passbands, "
                        "power-2 LD, eccentric)",
            "split_points_per_s": pts / (res["split"][0] / 1e3), "fp64_points_per_s": pts / (res["fp64"][0] / 1e3),
            "split_ms": res["split"][0], "fp64_ms": res["fp64"][0],
            "split_over_fp64": res["fp64"][0] / res["split"][0], "max_abs_dF_vs_fp64": dF,
            "fp64_culled_ms": res["fp64_culled"][0], "fp64_culled_same_bits": culled_same,
            "max_abs_dF_fp64_vs_oracle": float(np.abs(got64 - want).max()),
            "max_abs_dF_split_vs_oracle": float(np.abs(got32 - want).max()),
            "oracle_subset": f"{n_oracle} seeded parameter vectors x all {npt} times ({t_oracle:.1f} s on "
                             f"{os.cpu_count()} host threads)",
            "timed": "RoadRunnerModel.evaluate(copy=False), CUDA events, parameters uploaded each call"}


def bench_ts(torch, device, steps=20, npv=64, npb=200, npt=19700):
    """Transmission spectroscopy: 64 pv x 200 channels x 19,700 times (2-min
    cadence), quadratic LD, k ~ U(0.09, 0.11), one sample per point."""
    from pytransit_gb300 import TSModel
    rng = np.random.default_rng(4242)
    T = 2459000.0
    time_ = T + np.arange(npt) * (2.0 / 1440.0)
    a = rng.uniform(3.0, 20.0, npv)
    prm = dict(k=rng.uniform(0.09, 0.11, (npv, npb)),
               ldc=np.stack([rng.uniform(0, .6, (npv, npb)), rng.uniform(0, .3, (npv, npb))], -1),
               t0=T + 13.7 + rng.normal(0, 1e-3, npv), p=rng.uniform(0.5, 15.0, npv), a=a,
               i=np.arccos(rng.uniform(0.0, 0.9, npv) / a), e=np.zeros(npv), w=np.zeros(npv))
    res = {}
    models = {}
    for prec in ("split", "fp64"):
        m = models[prec] = TSModel('quadratic', precision=prec, device=device)
        m.set_data(time_)
        m.fp64_cull = False      # the plain FP64 path is the comparator
        res[prec] = bench_model(m, prm, steps if prec == "split" else 2, torch, device)
    # the drop-in's precision='fp64': the same FP64 arithmetic with the fold once per tile
    models["fp64"].fp64_cull = True
    res["fp64_culled"] = bench_model(models["fp64"], prm, 5, torch, device)
    culled_same = bool(torch.equal(res["fp64_culled"][1].nan_to_num(7.0), res["fp64"][1].nan_to_num(7.0)))
    dF = float((res["split"][1].double() - res["fp64"][1]).abs().max().item())
    pts = npv * npb * npt
    out_bytes = pts * 4
    peak, _ = measured_peaks()
    # host time of one evaluate() call (the calls are issued back to back;
    # the GPU work of a call overlaps the host work of the next)
    m = models["split"]
    argv = (prm["k"], prm["ldc"], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"], prm["w"])
    torch.cuda.synchronize(device)
    t = time.perf_counter()
    for _ in range(steps):
        m.evaluate(*argv, copy=False)
    host_ms = (time.perf_counter() - t) / steps * 1e3
    torch.cuda.synchronize(device)
    # the same model through the C ABI with its inputs resident in HBM:
    # the fused prologue and the flux kernel per step, CUDA events
    from pytransit_gb300 import _lib
    L = _lib.lib()
    P = _lib.ptr
    tb, dd = m._device_tables(device), m._device_data(device)
    dev = {n: torch.as_tensor(np.ascontiguousarray(prm[n], dtype=np.float64)).to(device)
           for n in ("k", "ldc", "t0", "p", "a", "i", "e", "w")}
    ldf = (npt + 3) // 4 * 4
    flux = torch.empty((npv, npb, ldf), dtype=torch.float32, device=device)
    wsb = L.rr_ts_workspace_bytes(1, npv, npb, m.ng)
    ws = torch.empty(wsb, dtype=torch.uint8, device=device)
    stream = torch.cuda.current_stream(device)
    sp = _lib.stream_ptr(device)
    orbit = tuple(P(dev[n]) for n in ("k", "t0", "p", "a", "i", "e", "w"))

    def step(ev=None):
        _lib.check(L.rr_ts_prepare_split_ld(m.ld_law, P(dev["ldc"]), 2, P(tb["mu"]), dd["t_ref"], dd["t_absmax"],
                                            *orbit, npv, npb, 0.0, m.ng, m.ze.size, P(tb["ze"]), P(ws), wsb, sp))
        if ev is not None:
            ev[0].record(stream)
        _lib.check(L.rr_ts_flux_split(P(dd["times_ff"]), npt, npv, npb, 1, 0.0, m.ng, m.dg, P(ws), P(flux), ldf, sp))
        if ev is not None:
            ev[1].record(stream)

    for _ in range(3):
        step()
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize(device)
    t0.record(stream)
    for j in range(steps):
        step(evs[j])
    t1.record(stream)
    torch.cuda.synchronize(device)
    dev_ms = t0.elapsed_time(t1) / steps
    flux_ms = statistics.mean(a.elapsed_time(b) for a, b in evs)
    dF_dev = float((flux[:, :, :npt].double() - res["fp64"][1]).abs().max().item())
    return {"workload": f"TSModel, {npv} pv x {npb} channels x {npt} times (2-min cadence), quadratic LD, nsamples=1",
            "split_points_per_s": pts / (res["split"][0] / 1e3), "fp64_points_per_s": pts / (res["fp64"][0] / 1e3),
            "split_ms": res["split"][0], "fp64_ms": res["fp64"][0],
            "split_over_fp64": res["fp64"][0] / res["split"][0], "max_abs_dF_vs_fp64": dF,
            "fp64_culled_ms": res["fp64_culled"][0], "fp64_culled_same_bits": culled_same,
            "split_output_gbs": out_bytes / (res["split"][0] / 1e3) / 1e9,
            "split_output_frac_of_hbm": out_bytes / (res["split"][0] / 1e3) / 1e9 / peak,
            "host_ms_per_call": host_ms,
            "timed": "TSModel.evaluate(copy=False) (prologue, 2D LD tables and flux), CUDA events, "
                     "parameters uploaded each call",
            "device_resident": {
                "ms_per_step": dev_ms, "points_per_s": pts / (dev_ms / 1e3),
                "output_frac_of_hbm": out_bytes / (dev_ms / 1e3) / 1e9 / peak,
                "flux_kernel_ms": flux_ms, "flux_kernel_frac_of_hbm": out_bytes / (flux_ms / 1e3) / 1e9 / peak,
                "max_abs_dF_vs_fp64": dF_dev,
                "timed": "rr_ts_prepare_split_ld + rr_ts_flux_split through the C ABI, inputs in HBM, CUDA events"}}


def bench_c3(torch, device, steps=10):
    """Log-likelihood + adjoint gradient, 4096 pv x 5000 times, 5 supersamples."""
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(77)
    npv, npt, sigma = 4096, 5000, 5e-4
    data = dict(time=np.linspace(-0.2, 0.2, npt), nsamples=[5], exptimes=[1 / 48])
    a0 = rng.uniform(3, 20)
    truth = dict(k=np.array([[rng.uniform(.05, .15)]]), ldc=np.array([[[rng.uniform(0, .6), rng.uniform(0, .3)]]]),
                 t0=np.array([[rng.normal(0, 1e-3)]]), p=np.array([rng.uniform(1, 10)]), a=np.array([a0]),
                 i=np.array([np.arccos(rng.uniform(0, .9) / a0)]), e=np.array([rng.uniform(0, .3)]),
                 w=np.array([rng.uniform(0, 2 * np.pi)]))
    m64 = RoadRunnerModel('quadratic', precision='fp64', device=device)
    m64.set_data(**data)
    f_true = m64.evaluate(truth["k"], truth["ldc"], truth["t0"], truth["p"], truth["a"], truth["i"], truth["e"],
                          truth["w"])
    obs = f_true + rng.normal(0, sigma, npt)
    prm = dict(k=truth["k"] * (1 + rng.normal(0, 0.02, (npv, 1))),
               ldc=np.clip(truth["ldc"] + rng.normal(0, 0.02, (npv, 1, 2)), 0.01, None),
               t0=truth["t0"] + rng.normal(0, 2e-4, (npv, 1)), p=truth["p"] * (1 + rng.normal(0, 1e-4, npv)),
               a=truth["a"] * (1 + rng.normal(0, 0.01, npv)), i=truth["i"] + rng.normal(0, 1e-3, npv),
               e=np.clip(truth["e"] + rng.normal(0, 0.01, npv), 0, None), w=truth["w"] + rng.normal(0, 0.05, npv))
    out = {}
    for prec in ("split", "fp64"):
        m = RoadRunnerModel('quadratic', precision=prec, device=device)
        m.set_data(**data)
        args = (m, obs, sigma, prm["k"], prm["ldc"], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"], prm["w"])
        lnlikelihood(*args, grad=True, copy=False)
        torch.cuda.synchronize(device)
        t = time.perf_counter()
        n = steps if prec == "split" else 2
        for _ in range(n):
            lnl, g = lnlikelihood(*args, grad=True, copy=False)
        torch.cuda.synchronize(device)
        out[prec] = ((time.perf_counter() - t) / n, lnl.cpu().numpy(), g.cpu().numpy())
    g32, g64 = out["split"][2], out["fp64"][2]
    col_rel = float((np.abs(g32 - g64) / np.abs(g64).max(axis=0, keepdims=True)).max())
    lnl_rel = float(np.abs(out["split"][1] - out["fp64"][1]).max() / np.abs(out["fp64"][1]).max())
    # central finite differences of the FP64 log-likelihood at the full size
    # (h = 1e-6 relative, with floors), element by element: |g - fd| against
    # 1e-4 |fd| plus the differences' own rounding floor (16 ulps of |lnL|
    # over the step), plus 1e-6 of the column's largest |fd| for the split path
    m64 = RoadRunnerModel('quadratic', precision='fp64', device=device)
    m64.set_data(**data)
    floors = dict(k=1e-3, t0=1e-2, p=1.0, a=1.0, i=1.0, e=1e-2, w=1e-1, ldc=1e-2)
    spec = [('k', (slice(None), 0)), ('t0', (slice(None), 0)), ('p', ()), ('a', ()), ('i', ()), ('e', ()),
            ('w', ()), ('ldc', (slice(None), 0, 0)), ('ldc', (slice(None), 0, 1))]

    def lnl64(q):
        return lnlikelihood(m64, obs, sigma, q["k"], q["ldc"], q["t0"], q["p"], q["a"], q["i"], q["e"], q["w"])

    base = {n: np.array(v, dtype=np.float64, copy=True) for n, v in prm.items()}
    lnl0 = np.abs(lnl64(base))

    def central(scale):
        fd_, fl_ = [], []
        for name, idx in spec:
            x = base[name][idx] if idx else base[name]
            h = scale * 1e-6 * np.maximum(np.abs(x), floors[name])
            up = {n: v.copy() for n, v in base.items()}
            dn = {n: v.copy() for n, v in base.items()}
            if idx:
                up[name][idx], dn[name][idx] = x + h, x - h
                step = up[name][idx] - dn[name][idx]
            else:
                up[name], dn[name] = x + h, x - h
                step = up[name] - dn[name]
            fd_.append((lnl64(up) - lnl64(dn)) / step)
            fl_.append(16 * np.finfo(np.float64).eps * lnl0 / step)
        return np.stack(fd_, -1), np.stack(fl_, -1)

    # the FD's uncertainty: its rounding, and its truncation (large where a step
    # crosses a kink of the piecewise-linear LD tables) as |FD(h) - FD(h/2)|
    fd_h, _ = central(0.01)
    fd, fl = central(0.005)
    fl = fl + np.abs(fd_h - fd)
    fd_check = {}
    # e = 0 (clipped) leaves no room for the step below: those elements have no central difference
    fin = np.isfinite(fd) & np.isfinite(fl)
    colmax = np.nanmax(np.where(fin, np.abs(fd), np.nan), axis=0, keepdims=True)
    for prec, g in (("fp64", g64), ("split", g32)):
        err = (np.abs(g - fd) / (1e-4 * np.abs(fd) + fl))[fin]
        big = fin & (np.abs(fd) > 100 * fl)
        fd_check[prec] = {"max_err_over_bound": float(err.max()), "elements_within_bound": float((err <= 1).mean()),
                          "max_rel_err_where_fd_above_100_floors": float((np.abs(g - fd)[big] / np.abs(fd)[big]).max()),
                          "max_abs_err_over_column_scale": float((np.abs(g - fd) / colmax)[fin].max())}
    fd_check["elements_without_central_difference"] = int((~fin).sum())
    # a repeated call gives the same bits (sums in a fixed order)
    msplit = RoadRunnerModel('quadratic', precision='split', device=device)
    msplit.set_data(**data)
    a1 = lnlikelihood(msplit, obs, sigma, prm["k"], prm["ldc"], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"],
                      prm["w"], grad=True)
    a2 = lnlikelihood(msplit, obs, sigma, prm["k"], prm["ldc"], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"],
                      prm["w"], grad=True)
    reproducible = bool(np.array_equal(a1[0], a2[0]) and np.array_equal(a1[1], a2[1]))
    return {"workload": f"{npv} pv x {npt} times, 5 supersamples, quadratic LD, Gaussian lnL sigma=5e-4, "
                        "gradient wrt (k, t0, p, a, i, e, w, u1, u2)",
            "split_ms": out["split"][0] * 1e3, "fp64_ms": out["fp64"][0] * 1e3,
            "split_points_per_s": npv * npt / out["split"][0], "fp64_points_per_s": npv * npt / out["fp64"][0],
            "split_over_fp64": out["fp64"][0] / out["split"][0],
            "grad_max_rel_err_split_vs_fp64": col_rel, "lnl_max_rel_err_split_vs_fp64": lnl_rel,
            "grad_vs_fd": dict(fd_check, what="per element: |g - fd| / (1e-4 |fd| + floor) <= 1 is within the "
                                              "1e-4 relative target; FD of the FP64 lnL, h = 5e-9 relative; floor = "
                                              "16 ulps of |lnL| / step + |FD(2h) - FD(h)|"),
            "bit_reproducible": reproducible,
            "timed": "lnlikelihood(grad=True) end to end (LD tables, prologue, fused lnL + adjoint), wall clock"}


def bench_eclipse(torch, device, data, prm, steps=3):
    """The secondary-eclipse model on the default workload's data and
    population (8192 pv x 19,700 times), FP64 and split: model points/s
    (CUDA events, parameters uploaded each call) and the split path's max
    |dF| against FP64."""
    from pytransit_gb300 import EclipseModel
    args = (prm["k"][:, 0], prm["t0"], prm["p"], prm["a"], prm["i"], prm["e"], prm["w"])
    res, outs = {}, {}
    # the split leg first: little else is held on the device while it runs
    for prec, n in (("split", 10 * steps), ("fp64", steps), ("fp64_culled", steps)):
        m = EclipseModel(precision="split" if prec == "split" else "fp64", device=device)
        m.fp64_cull = prec == "fp64_culled"      # the plain FP64 path is the comparator
        m.set_data(data["time"], lcids=data["lcids"], pbids=data["pbids"])
        m.evaluate(*args, copy=False)
        stream = torch.cuda.current_stream(device)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize(device)
        e0.record(stream)
        for _ in range(n):
            out = m.evaluate(*args, copy=False)
        e1.record(stream)
        torch.cuda.synchronize(device)
        res[prec] = e0.elapsed_time(e1) / n
        outs[prec] = out
    # the split step through the C ABI with the parameters already in HBM
    from pytransit_gb300 import _lib
    from pytransit_gb300.eclipse import _L
    m = EclipseModel(precision='split', device=device)
    m.set_data(data["time"], lcids=data["lcids"], pbids=data["pbids"])
    dd = m._device_data(device)
    npv = prm["p"].size
    g = m._upload(dict(k=np.ascontiguousarray(prm["k"][:, 0]), t0=prm["t0"], p=prm["p"], a=prm["a"], i=prm["i"],
                       e=prm["e"], w=prm["w"], rstar=np.ones(npv)), device)
    L, P = _L(), _lib.ptr
    wsb = L.rr_eclipse_split_workspace_bytes(npv, m.nlc, 1)
    ws = torch.empty(wsb, dtype=torch.uint8, device=device)
    dev_out = torch.empty((npv, m.npt), dtype=torch.float32, device=device)
    stream = torch.cuda.current_stream(device)

    def step():
        _lib.check(L.rr_eclipse_split(P(dd['times_ff']), dd['t_ref'], dd['t_absmax'], m.npt, P(g['k']), P(g['t0']),
                                      1, P(g['p']), P(g['a']), P(g['i']), P(g['e']), P(g['w']), P(g['rstar']), npv,
                                      m.nlc, P(dd['lcids']), P(dd['epids']), P(dd['nsamples']), P(dd['exptimes']),
                                      P(ws), wsb, P(dev_out), m.npt, _lib.stream_ptr(device)), "rr_eclipse_split")
    for _ in range(3):
        step()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize(device)
    e0.record(stream)
    for _ in range(20):
        step()
    e1.record(stream)
    torch.cuda.synchronize(device)
    dev_ms = e0.elapsed_time(e1) / 20
    peak, _ = measured_peaks()
    k2 = torch.as_tensor(np.pi * prm["k"][:, :1] ** 2).to(device)
    npts = outs["fp64"].numel()
    dmax = float((outs["split"].double() - outs["fp64"]).abs().max().item())
    return {"workload": "EclipseModel.evaluate(copy=False), 8192 pv x 19700 times, parameters uploaded each call, "
                        "CUDA events", "points_per_s": npts / (res["fp64"] * 1e-3), "ms": res["fp64"],
            "split_points_per_s": npts / (res["split"] * 1e-3), "split_ms": res["split"],
            "split_over_fp64": res["fp64"] / res["split"], "max_abs_dF_split_vs_fp64": dmax,
            "fp64_culled_ms": res["fp64_culled"],
            "fp64_culled_same_bits": bool(torch.equal(outs["fp64_culled"].nan_to_num(7.0), outs["fp64"].nan_to_num(7.0))),
            "split_device_resident": {"ms_per_step": dev_ms, "points_per_s": npts / (dev_ms * 1e-3),
                                      "output_frac_of_hbm": 4.0 * npts / (dev_ms * 1e-3) / (peak * 1e9),
                                      "timed": "rr_eclipse_split (prologue + flux) through the C ABI, inputs in "
                                               "HBM, CUDA events"},
            "in_eclipse_fraction": float((outs["fp64"] < k2 - 1e-12).double().mean().item())}


class C4Mix:
    """The serving mix: npv log-uniform [1, 4096], npt log-uniform [500, 1e5],
    nsamples in {1, 5, 10}, LD in {quadratic, power-2, nonlinear}, 20 %
    transmission-spectroscopy requests with 200 channels, k ~ U(0.09, 0.11);
    2-min cadence from BJD 2459000.  Requests are views into shared pools
    (times, radius ratios, LD coefficients), so that thousands of them cost
    no host memory or generation time."""
    LDC = {'quadratic': [0.35, 0.15], 'power-2': [0.6, 0.55], 'nonlinear': [0.5, -0.2, 0.6, -0.25]}

    def __init__(self, seed=4):
        pool = np.random.default_rng(1000 + seed)
        self.rng = np.random.default_rng(seed)
        self.time = 2459000.0 + np.arange(100000) * (2 / 1440)
        self.k_ts = pool.uniform(0.09, 0.11, (2 * 4096, 200))
        self.k_rr = pool.uniform(0.05, 0.15, (2 * 4096, 1))
        self.ldc = {law: np.ascontiguousarray(np.broadcast_to(np.asarray(v, np.float64), (4096, 200, len(v))))
                    for law, v in self.LDC.items()}

    def request(self):
        rng = self.rng
        T = 2459000.0
        kind = 'ts' if rng.uniform() < 0.2 else 'rr'
        law = ['quadratic', 'power-2', 'nonlinear'][int(rng.integers(0, 3))]
        npv = int(np.exp(rng.uniform(0, np.log(4096))))
        npt = int(np.exp(rng.uniform(np.log(500), np.log(1e5))))
        ns = int(rng.choice([1, 5, 10]))
        cad = 2 / 1440
        npb = 200 if kind == 'ts' else 1
        o = int(rng.integers(0, 4096))
        k = (self.k_ts if kind == 'ts' else self.k_rr)[o:o + npv]
        a = rng.uniform(3, 20, npv)
        params = dict(k=k, ldc=self.ldc[law][:npv, :npb], t0=T + rng.normal(0, 1e-3, npv),
                      p=rng.uniform(0.5, 15, npv), a=a, i=np.arccos(rng.uniform(0, 0.9, npv) / a),
                      e=np.zeros(npv), w=np.zeros(npv))
        data = dict(time=self.time[:npt], nsamples=[ns], exptimes=[cad if ns > 1 else 0.0])
        return kind, law, data, params


def serve_run(srv, reqs, rate, seed=5):
    """Submit reqs as a Poisson stream at `rate` requests/s; wait for all.
    Returns the run's figures (latencies from submit to resolve)."""
    rng = np.random.default_rng(seed)
    gaps = rng.exponential(1.0 / rate, len(reqs))
    st0 = dict(srv.stats.summary())
    lat0 = len(srv.stats.latencies)
    futs = []
    t_start = time.perf_counter()
    t_next = t_start
    for r, gap in zip(reqs, gaps):
        t_next += gap
        while time.perf_counter() < t_next:
            time.sleep(0.0001)
        futs.append((time.perf_counter(), srv.submit(*r, keep_result=False)))
    t_arrivals = time.perf_counter()
    load_end = srv.load()
    points, done, rejected, failed = 0, [], 0, 0
    for t_sub, f in futs:
        try:
            points += f.result()
            done.append(t_sub)
        except MemoryError:
            rejected += 1
        except Exception:
            failed += 1
    t_end = time.perf_counter()
    st = srv.stats.summary()
    lat = np.array(srv.stats.latencies[lat0:])
    dts = np.array(srv.stats.done_times[lat0:])
    n = len(lat)
    half = n // 2
    p99 = lambda x: float(np.percentile(x, 99)) if len(x) else None
    in_window = int((dts <= t_arrivals).sum()) if n else 0
    wall_arr = t_arrivals - t_start
    return {"offered_req_per_s": rate, "requests": len(reqs), "completed": n, "rejected": rejected,
            "failed": failed, "arrival_window_s": wall_arr, "wall_s": t_end - t_start,
            "achieved_req_per_s": n / (t_end - t_start),
            "completed_in_window_req_per_s": in_window / wall_arr,
            "points_per_s": points / (t_end - t_start),
            "latency_p50_s": float(np.percentile(lat, 50)) if n else None, "latency_p99_s": p99(lat),
            "latency_mean_s": float(lat.mean()) if n else None,
            "latency_p99_first_half_s": p99(lat[:half]), "latency_p99_second_half_s": p99(lat[half:]),
            "queued_at_end_of_arrivals": load_end["queued"], "active_at_end_of_arrivals": load_end["active"],
            "admitted_bytes_at_end_of_arrivals": load_end["admitted_bytes"],
            "steps": st["steps"] - st0["steps"], "bypassed": st["bypassed"] - st0["bypassed"],
            # where the wall time went: device time of the batched steps, and
            # the scheduler thread's time in admission + set-up, step issue and
            # completion polling
            "gpu_step_busy": (st["gpu_step_s"] - st0["gpu_step_s"]) / (t_end - t_start),
            "host_admit_busy": (st["admit_s"] - st0["admit_s"]) / (t_end - t_start),
            "host_step_busy": (st["step_s"] - st0["step_s"]) / (t_end - t_start),
            "host_poll_busy": (st["poll_s"] - st0["poll_s"]) / (t_end - t_start)}


def sustained(run):
    """Achieved = offered, the queue empty when arrivals stop, p99 flat."""
    a, b = run["latency_p99_first_half_s"], run["latency_p99_second_half_s"]
    return (run["achieved_req_per_s"] >= 0.97 * run["offered_req_per_s"] and
            run["queued_at_end_of_arrivals"] <= max(10, 0.01 * run["requests"]) and
            a is not None and b is not None and b <= 1.5 * a + 0.005)


def per_request_paths(reqs, torch, device, nsample):
    """The first nsample requests one at a time through the drop-in models
    (no batching): the plain FP64 path, and the split path beside it.  A
    request larger than the server's budget (which the server rejects) or
    whose FP64 output would take more than 100 GB is skipped."""
    from pytransit_gb300 import RoadRunnerModel, TransmissionSpectroscopyModel
    out, models = {}, {}
    for prec in ("fp64", "split"):
        n, t_tot, pts, skipped = 0, 0.0, 0, 0
        for kind, law, data, params in reqs[:nsample]:
            npv, npt = params["p"].size, data["time"].size
            npb = params["k"].shape[1] if kind == 'ts' else 1
            if npv * npb * npt * 4 > 120e9 or npv * npb * npt * 8 > 100e9:
                skipped += 1
                continue
            key = (kind, law, prec)
            if key not in models:
                M = TransmissionSpectroscopyModel if kind == 'ts' else RoadRunnerModel
                models[key] = M(law, precision=prec, device=device)
                models[key].fp64_cull = False      # the plain FP64 path per request is the comparator
            m = models[key]
            if kind == 'ts':
                m.set_data(data["time"], nsamples=data["nsamples"], exptimes=data["exptimes"])
                argv = (params["k"], params["ldc"], params["t0"], params["p"], params["a"], params["i"],
                        params["e"], params["w"])
            else:
                m.set_data(**data)
                argv = (params["k"], params["ldc"], params["t0"].reshape(-1, 1), params["p"], params["a"],
                        params["i"], params["e"], params["w"])
            torch.cuda.synchronize(device)
            t = time.perf_counter()
            res = m.evaluate(*argv, copy=False)
            torch.cuda.synchronize(device)
            t_tot += time.perf_counter() - t
            pts += res.numel()
            n += 1
            del res
        out[prec] = dict(requests=n, skipped=skipped, points_per_s=pts / max(t_tot, 1e-9), wall_s=t_tot)
    del models
    torch.cuda.empty_cache()
    return out


def serve_suite(torch, device, rate=2000.0, duration_s=5.0, probe_s=2.5, max_probes=3, plain_sample=200):
    """The serving leg: the C4 mix as a Poisson stream at `rate` for
    `duration_s` through RRServer (split precision, device-resident results,
    120 GB budget); then shorter runs at other rates to find the highest one
    the server sustains (upwards in 1.5x steps if `rate` is sustained, else
    downwards); then the plain FP64 path on the same requests one at a time."""
    from pytransit_gb300.serving import RRServer
    mix = C4Mix(4)
    srv = RRServer(hbm_budget=120e9, result='device', device=device)
    srv.submit(*C4Mix(99).request(), keep_result=False).result()      # warm-up: tables, graph, arena
    reqs = [mix.request() for _ in range(int(rate * duration_s))]
    with ClockSampler(0) as clk:
        main_run = serve_run(srv, reqs, rate)
    clocks = clk.summary()
    probes = []
    ok = sustained(main_run)
    lo, hi = (rate, None) if ok else (None, rate)     # highest sustained / lowest not sustained so far
    for j in range(max_probes):
        if lo is not None and hi is not None:
            r = (lo * hi) ** 0.5                        # bisect (geometrically) once bracketed
        else:
            r = lo * 1.5 if hi is None else hi / 1.5
        run = serve_run(srv, [mix.request() for _ in range(int(r * probe_s))], r, seed=6 + j)
        probes.append({k: run[k] for k in ("offered_req_per_s", "achieved_req_per_s", "latency_p50_s",
                                            "latency_p99_s", "latency_p99_first_half_s",
                                            "latency_p99_second_half_s", "queued_at_end_of_arrivals",
                                            "points_per_s", "gpu_step_busy", "host_admit_busy",
                                            "host_step_busy", "host_poll_busy")})
        good = sustained(run)
        probes[-1]["sustained"] = good
        if good:
            lo = r if lo is None else max(lo, r)
        else:
            hi = r if hi is None else min(hi, r)
    best = lo
    srv.close()
    plain = per_request_paths(reqs, torch, device, plain_sample)
    res = dict(main_run)
    res.update({
        "workload": f"C4 mix, Poisson arrivals at {rate:g} req/s for {duration_s:g} s ({len(reqs)} requests): npv "
                    "log-U[1,4096], npt log-U[500,1e5], nsamples {1,5,10}, LD {quadratic, power-2, nonlinear}, "
                    "20% TS with 200 channels; split precision; results kept on the device; HBM budget 120 GB",
        "sustained": ok, "max_sustained_req_per_s": best, "lowest_unsustained_req_per_s": hi,
        "rate_probes": probes,
        "plain_fp64_per_request": dict(plain["fp64"], sample=f"the first {plain_sample} requests of the stream one "
                                       "at a time, RoadRunnerModel / TransmissionSpectroscopyModel precision='fp64', "
                                       "copy=False, data upload included"),
        "split_per_request": dict(plain["split"], sample="the same requests one at a time, precision='split'"),
        "served_over_plain_fp64": main_run["points_per_s"] / plain["fp64"]["points_per_s"],
        "clocks": clocks})
    return res


def bench_serve(args):
    """--workload serve: the serving leg alone, one JSON line."""
    import torch
    device = torch.device("cuda", 0)
    torch.cuda.set_device(device)
    res = serve_suite(torch, device, rate=args.rate, duration_s=args.serve_s, plain_sample=args.plain_sample,
                      max_probes=args.probes)
    line = {"metric": "served model points/s (Poisson request stream); p50/p99 latency",
            "value": res["points_per_s"], "unit": "model points/s", "n_gpus": 1, "higher_is_better": True,
            "data": "synthetic (seeded)", "config": {"workload": res["workload"]}, **res}
    print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--npv", type=int, default=8192)
    ap.add_argument("--npt", type=int, default=19700)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-parity", action="store_true", help="skip the full-size check against the oracle")
    ap.add_argument("--no-serve", action="store_true", help="skip the serving leg of the default line")
    ap.add_argument("--no-extra", action="store_true", help="skip the precision and gradient workloads")
    ap.add_argument("--workload", default="c1", choices=["c1", "c2", "c3", "ts", "eclipse", "serve"],
                    help="c1: the default line; c2 / c3 / ts / eclipse: the precision / gradient / "
                         "transmission-spectroscopy / secondary-eclipse workload alone; serve: Poisson stream")
    ap.add_argument("--rate", type=float, default=2000.0, help="serving leg: offered requests/s")
    ap.add_argument("--serve-s", type=float, default=5.0, help="serving leg: seconds of arrivals at --rate")
    ap.add_argument("--plain-sample", type=int, default=200,
                    help="serving leg: requests run one at a time through the plain FP64 path")
    ap.add_argument("--probes", type=int, default=3,
                    help="serving leg: runs at other rates that bracket the highest sustained rate")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        return impl_reference(args, rank)
    if args.workload == "serve":
        return bench_serve(args) if rank == 0 else 0
    if args.workload in ("c2", "c3", "ts", "eclipse"):
        if rank == 0:
            import torch
            device = torch.device("cuda", 0)
            torch.cuda.set_device(device)
            if args.workload == "eclipse":
                res = bench_eclipse(torch, device, *workload(args.npv, args.npt))
            else:
                res = {"c2": bench_c2, "c3": bench_c3, "ts": bench_ts}[args.workload](torch, device)
            print(json.dumps({"workload": args.workload, **res}), flush=True)
        return 0

    import torch
    import torch.distributed as dist
    from pytransit_gb300 import RoadRunnerModel, _lib

    torch.cuda.set_device(local_rank)
    device = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=device)

    from pytransit_gb300.sharding import barrier, max_over_ranks

    # Each rank evaluates its own population (weak scaling, no collective on the data path).
    data, prm = workload(args.npv, args.npt, seed=1234 + rank)
    npv, npt = args.npv, args.npt
    model = RoadRunnerModel('quadratic', precision='split', device=device)
    model.set_data(**data)
    dd = model._device_data(device)
    tb = model._device_tables(device)
    L = _lib.lib()
    stream = torch.cuda.current_stream(device)
    sp = _lib.stream_ptr(device)
    nz, ng, nk = model.ze.size, model.ng, model.nk
    nlc, npb, nep = model.nlc, model.npb, 1
    dev = {n: torch.as_tensor(np.ascontiguousarray(v)).to(device) for n, v in prm.items()}
    ldp32 = torch.empty((npv, npb, nz), dtype=torch.float32, device=device)
    ist32 = torch.empty((npv, npb), dtype=torch.float32, device=device)
    ldp64 = torch.empty((npv, npb, nz), dtype=torch.float64, device=device)
    ist64 = torch.empty((npv, npb), dtype=torch.float64, device=device)
    ldf = (npt + 3) // 4 * 4
    flux32 = torch.empty((npv, ldf), dtype=torch.float32, device=device)
    flux64 = torch.empty((npv, npt), dtype=torch.float64, device=device)
    ws32 = torch.empty(L.rr_full_split_workspace_bytes(npv, npb, nlc, nep, ng), dtype=torch.uint8, device=device)
    ws64 = torch.empty(L.rr_full_f64_workspace_bytes(npv, npb, ng), dtype=torch.uint8, device=device)
    P = _lib.ptr
    kmin, kmax = float(model.klims[0]), float(model.klims[1])
    B32, nb = model._basis(device, 2, True)
    B64, _ = model._basis(device, 2, False)

    def step_split(ev=None):
        _lib.check(L.rr_prepare_split_ld(dd["t_ref"], dd["t_absmax"], P(dev["k"]), 1, P(dev["t0"]), 1, nep,
                                         P(dev["p"]), P(dev["a"]), P(dev["i"]), P(dev["e"]), P(dev["w"]), npv,
                                         nlc, npb, P(dd["pbids"]), P(dd["epids"]), P(dd["nsamples"]),
                                         P(dd["exptimes"]), 2, P(dev["ldc"]), 2, P(tb["mu"]), nz, P(B32), nb,
                                         P(tb["W32"]), nk, ng, model.dk, kmin, kmax, P(tb["ze"]), P(ldp32),
                                         P(ist32), P(ws32), ws32.numel(), sp))
        if ev is not None:
            ev[0].record(stream)
        _lib.check(L.rr_flux_split_rows(P(dd["times_ff"]), npt, P(dd["lcids"]), npv, nlc, npb, ng, model.dg,
                                        P(ws32), 0, npv, P(flux32), ldf, dd["rows"], sp))
        if ev is not None:
            ev[1].record(stream)

    def step_fp64():
        _lib.check(L.rr_ld_tables_f64(2, P(dev["ldc"]), npv, npb, 2, P(tb["mu"]), nz, P(ldp64), P(ist64), sp))
        _lib.check(L.rr_prepare_f64(P(dev["k"]), 1, P(dev["p"]), P(dev["a"]), P(dev["i"]), P(dev["e"]),
                                    P(dev["w"]), npv, npb, P(ldp64), P(tb["W64"]), nk, ng, nz, model.dk, kmin, kmax,
                                    P(tb["ze"]), P(ws64), ws64.numel(), sp, 2, P(dev["ldc"]), 2, P(B64), nb))
        _lib.check(L.rr_flux_f64(P(dd["time"]), npt, P(dev["k"]), 1, P(dev["t0"]), 1, P(dev["p"]), npv, nlc, npb,
                                 P(dd["lcids"]), P(dd["pbids"]), P(dd["epids"]), P(dd["nsamples"]),
                                 P(dd["exptimes"]), P(ist64), ng, model.dg, P(ws64), P(flux64), npt, sp))

    def timed(fn, steps, warmup, per_step_events=False):
        gc.collect()   # a collection of the imported modules' objects takes about eight steps
        for _ in range(warmup):
            fn()
        barrier()
        torch.cuda.synchronize(device)
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
               for _ in range(steps)] if per_step_events else None
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        for s in range(steps):
            if per_step_events:
                fn(evs[s])
            else:
                fn()
        t1.record(stream)
        torch.cuda.synchronize(device)
        barrier()
        ms = t0.elapsed_time(t1)
        kern = [a.elapsed_time(b) for a, b in evs] if per_step_events else None
        return ms, kern

    # --- split path, device-resident inputs (the headline `value`) ---
    with ClockSampler(local_rank) as clk:
        ms_split, kern_ms = timed(step_split, args.steps, args.warmup, per_step_events=True)
    clocks = clk.summary()
    ms_split = max_over_ranks(ms_split)
    per_step_s = ms_split / 1e3 / args.steps
    value = world * npv * npt / per_step_s

    # --- plain FP64 path ---
    fp64_steps = max(3, args.steps // 4)
    ms64, _ = timed(step_fp64, fp64_steps, 2)
    ms64 = max_over_ranks(ms64)
    value64 = world * npv * npt / (ms64 / 1e3 / fp64_steps)

    # --- the drop-in's FP64 precision: the same arithmetic with the fold once
    # per tile for tiles that reach no box (identical bits) ---
    flux64c = torch.empty_like(flux64)

    def step_fp64_culled():
        _lib.check(L.rr_ld_tables_f64(2, P(dev["ldc"]), npv, npb, 2, P(tb["mu"]), nz, P(ldp64), P(ist64), sp))
        _lib.check(L.rr_prepare_f64(P(dev["k"]), 1, P(dev["p"]), P(dev["a"]), P(dev["i"]), P(dev["e"]),
                                    P(dev["w"]), npv, npb, P(ldp64), P(tb["W64"]), nk, ng, nz, model.dk, kmin, kmax,
                                    P(tb["ze"]), P(ws64), ws64.numel(), sp, 2, P(dev["ldc"]), 2, P(B64), nb))
        _lib.check(L.rr_flux_f64_culled_range(P(dd["time"]), P(dd["tiles64"]), npt, P(dev["k"]), 1, P(dev["t0"]), 1,
                                              P(dev["p"]), npv, nlc, npb, P(dd["lcids"]), P(dd["pbids"]),
                                              P(dd["epids"]), P(dd["nsamples"]), P(dd["exptimes"]), P(ist64), ng,
                                              model.dg, P(ws64), 0, npv, P(flux64c), npt, sp))

    ms64c, _ = timed(step_fp64_culled, args.steps, 2)
    ms64c = max_over_ranks(ms64c)

    # accuracy of the split path on this workload, full size (max |dF| vs FP64)
    step_split()
    step_fp64()
    torch.cuda.synchronize(device)
    culled_same = bool(torch.equal(flux64c.nan_to_num(7.0), flux64.nan_to_num(7.0)))
    del flux64c
    dF = float((flux32[:, :npt].double() - flux64).abs().max().item())
    in_transit = float((flux64 < 1.0).double().mean().item())
    # host copies of both results, checked against the oracle's FP64 flux of the
    # whole population after the CPU-baseline leg has computed it
    host64 = flux64.cpu().numpy() if rank == 0 and world == 1 and not args.no_parity else None
    host32 = flux32[:, :npt].cpu().numpy() if host64 is not None else None
    # independent cross-check: the Mandel & Agol quadratic model on the same
    # orbit layer as the FP64 RoadRunner step just run (its workspace)
    ma_check = None
    if not args.no_extra:
        from pytransit_gb300 import crosscheck
        fma = torch.empty_like(flux64)
        _lib.check(crosscheck._L().rr_ma_quad_flux_f64(
            P(dd["time"]), npt, P(dev["k"]), 1, P(dev["t0"]), 1, P(dev["p"]), npv, nlc, npb, P(dd["lcids"]),
            P(dd["pbids"]), P(dd["epids"]), P(dd["nsamples"]), P(dd["exptimes"]), P(dev["ldc"]), P(ws64), P(fma),
            npt, sp), "rr_ma_quad_flux_f64")
        ma_check = {"max_abs_dF_roadrunner_vs_mandel_agol": float((flux64 - fma).abs().max().item()),
                    "what": "plain FP64 RoadRunner vs the Mandel & Agol quadratic model (elliptic integrals) on "
                            "the same orbit, fold and bounding box, whole workload: RoadRunner's discretisation"}
        del fma

    # --- end to end through the public API: host params in, pinned host flux out ---
    host_out = torch.empty((npv, npt), dtype=torch.float32, pin_memory=True)
    e2e_prm = {n: np.ascontiguousarray(v) for n, v in prm.items()}

    def step_e2e():
        model.evaluate(e2e_prm["k"], e2e_prm["ldc"], e2e_prm["t0"], e2e_prm["p"], e2e_prm["a"],
                       e2e_prm["i"], e2e_prm["e"], e2e_prm["w"], out=host_out)

    def timed_e2e():
        for _ in range(args.warmup):
            step_e2e()
        barrier()
        torch.cuda.synchronize(device)
        t = time.perf_counter()
        for _ in range(e2e_steps):
            step_e2e()
        torch.cuda.synchronize(device)
        return max_over_ranks(time.perf_counter() - t) / e2e_steps

    e2e_steps = max(3, args.steps // 2)
    # the whole flux copied over in chunks (the host link carries all 4 B per point)
    model.host_fill = False
    e2e_copy_s = timed_e2e()
    copy_ok = bool(torch.equal(host_out, flux32[:, :npt].cpu()))
    # the default: the host sets the rows to 1 while the GPU writes the transit tiles into them
    model.host_fill = True
    e2e_s = timed_e2e()
    fill_ok = bool(torch.equal(host_out, flux32[:, :npt].cpu()))
    e2e_value = world * npv * npt / e2e_s
    h2d = sum(v.size for v in prm.values()) * 8
    # bytes the GPU writes into host memory per step: the tiles that reach a
    # transit window (counted once, on a device buffer holding a sentinel)
    sent = torch.full((npv, npt), -3.0, dtype=torch.float32, device=device)
    _lib.check(L.rr_flux_split_transits(P(dd["times_ff"]), npt, P(dd["lcids"]), npv, nlc, npb, ng, model.dg,
                                        P(ws32), 0, npv, P(sent), npt, sp), "rr_flux_split_transits")
    ncopy = int(round(npv * (1.0 - model.host_fill_fraction)))
    d2h = ncopy * npt * 4 + int((sent[ncopy:] != -3.0).sum().item()) * 4
    del sent

    # the drop-in's default call, evaluate(...) -> numpy float64 (copy=True),
    # in both precisions: what a user of the reference gets by swapping the
    # class; the result of each call is released before the next (as a
    # sampler loop does), so the pinned host buffer is reused
    def default_call(m):
        out = None
        for _ in range(2):
            out = m.evaluate(*(e2e_prm[n] for n in ("k", "ldc", "t0", "p", "a", "i", "e", "w")))
        del out
        ts = []
        for _ in range(max(3, e2e_steps // 2)):
            t = time.perf_counter()
            out = m.evaluate(*(e2e_prm[n] for n in ("k", "ldc", "t0", "p", "a", "i", "e", "w")))
            ts.append(time.perf_counter() - t)
            del out
        return statistics.median(ts)

    dc_split = default_call(model)
    model64 = RoadRunnerModel('quadratic', device=device)
    model64.set_data(**data)
    dc_fp64 = default_call(model64)
    del model64

    # --- roofline of the flux kernel ---
    kern_avg_s = statistics.mean(kern_ms) / 1e3
    s_out, s_tab = 4, 4
    bytes_alg = (npv * npt * s_out + npt * (8 + 4) + npv * npb * (ng + 1) * s_tab
                 + npv * (10 * 8 + nlc * 16))
    achieved = bytes_alg / kern_avg_s / 1e9
    peak, peak_kind = measured_peaks()
    traffic = profiled_traffic(npv, npt)

    line = {
        "metric": METRIC, "value": value, "unit": "model points/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": per_step_s * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32 per-sample arithmetic, f64 orbit/phase data (split precision)",
        "data": "synthetic (seeded; no public dataset)",
        "config": {"workload": WORKLOAD, "npv_per_gpu": npv, "npt": npt, "npb": npb, "nlc": nlc,
                   "nsamples": 1, "ld": "quadratic", "precision": "split",
                   "l2": "no flush: each step writes npv*npt*4 B of flux (645 MB > 129 MB L2)",
                   "parallelism": f"replicas x{world} (independent populations per GPU)"},
        "fp64_path": {"value": value64, "unit": "model points/s", "ms_per_step": ms64 / fp64_steps,
                      "what": "plain all-FP64 GPU path: every point through the reference's FP64 arithmetic "
                              "(rr_flux_f64), the comparator the metric names"},
        "fp64_culled_path": {"value": world * npv * npt / (ms64c / 1e3 / args.steps), "unit": "model points/s",
                             "ms_per_step": ms64c / args.steps, "same_bits_as_plain": culled_same,
                             "what": "the drop-in's precision='fp64': the same FP64 arithmetic, the fold once per "
                                     "128-point tile for tiles that reach no box (rr_flux_f64_culled_range)"},
        "split_over_fp64": value / value64,
        "max_abs_dF_vs_fp64": dF,
        "mandel_agol_crosscheck": ma_check,
        "in_transit_fraction": in_transit,
        "e2e": {"value": e2e_value, "unit": "model points/s", "h2d_bytes_per_step": int(h2d),
                "d2h_bytes_per_step": int(d2h), "ms_per_step": e2e_s * 1e3,
                "path": "RoadRunnerModel.evaluate(numpy params, out=pinned host float32)",
                "output": f"{1 - model.host_fill_fraction:.2f} of the rows computed on the device and copied "
                          f"over; meanwhile {model.host_threads} host threads set the other rows to 1, a pv chunk "
                          "at a time, and the GPU writes each chunk's tiles that reach a transit window straight "
                          "into the pinned rows (d2h_bytes_per_step counts both); the result equals the "
                          "device-resident flux bit for bit",
                "equals_device_result": fill_ok,
                "default_call": {"path": "RoadRunnerModel(...).evaluate(numpy params) -> numpy float64 "
                                         "(copy=True, the reference's signature and return type)",
                                 "split_ms": dc_split * 1e3, "split_points_per_s": npv * npt / dc_split,
                                 "fp64_ms": dc_fp64 * 1e3, "fp64_points_per_s": npv * npt / dc_fp64,
                                 "d2h_bytes_per_call_fp64": npv * npt * 8},
                "copy_path": {"value": world * npv * npt / e2e_copy_s, "ms_per_step": e2e_copy_s * 1e3,
                              "d2h_bytes_per_step": npv * npt * 4, "equals_device_result": copy_ok,
                              "path": "the same call with host_fill=False: the whole flux computed on the "
                                      "device and copied to the pinned rows in chunks"}},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": traffic, "peak_kind": peak_kind,
                     "kernel": "flux_split_kernel", "kernel_ms": kern_avg_s * 1e3,
                     "bytes_alg_per_launch": bytes_alg,
                     # the same kernel time against the DRAM bytes ncu measured for it: part of the
                     # algorithmic bytes (LD tables, the output's tail) are served by or stay in L2
                     "achieved_dram": traffic / kern_avg_s / 1e9 if traffic else None,
                     "frac_dram": traffic / kern_avg_s / 1e9 / peak if traffic else None},
        "clocks": clocks,
        # per step: the fused prologue (LD tables, LD means, orbit records) and the flux kernel
        "gpu_launches": 2 * args.steps,
    }
    if rank == 0 and not args.no_extra:
        line["c2_precision"] = bench_c2(torch, device)
        line["c3_gradient"] = bench_c3(torch, device)
        line["ts"] = bench_ts(torch, device)
        line["eclipse"] = bench_eclipse(torch, device, data, prm)
    if rank == 0 and world == 1 and not args.no_serve:
        del flux64, flux32, ws32, ws64
        torch.cuda.empty_cache()
        line["serve"] = serve_suite(torch, device, rate=args.rate, duration_s=args.serve_s,
                                    plain_sample=args.plain_sample, max_probes=args.probes)
    keep = {}
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = run_cpu_baseline(data, prm, keep=keep)
    if host64 is not None:
        if "flux" not in keep:
            keep["flux"] = cpu_rr_full(cpu_oracle_model(data), prm, npv, os.cpu_count() or 1)
        want = keep.pop("flux")
        line["parity_vs_oracle"] = {
            "max_abs_dF_fp64_vs_oracle": float(np.abs(host64 - want).max()),
            "max_abs_dF_split_vs_oracle": float(np.abs(host32.astype(np.float64) - want).max()),
            "points": int(want.size), "bound_fp64": 1e-9, "bound_split": 1e-6,
            "what": "the whole workload (all parameter vectors x all times): the GPU's FP64 and split results "
                    "against the oracle's FP64 rr_full restatement (oracle/rr_oracle.c) on the host cores"}
        del want, host64, host32
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
