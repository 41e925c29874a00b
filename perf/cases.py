"""Performance cases of the transit-model framework: what a user's program has it do.

Five families, each through its public entry points:

* ``rr``: RoadRunnerModel.evaluate, one optimiser call up to whole populations;
* ``ts``: TransmissionSpectroscopyModel.evaluate, wavelength channels sharing an orbit;
* ``ecl``: EclipseModel.evaluate and EclipseSpectroscopyModel.evaluate;
* ``lnl``: the Gaussian log-likelihood, forward (sampler populations on the
  device) and with its adjoint (autograd);
* ``serve``: a burst of mixed requests through RRServer.

``exact`` restates the same discretised model (weight table, LD means, Taylor
orbit, box, kite area) in plain torch FP64.
"""
import math

import numpy as np
import torch

T_BJD = 2459000.0          # BJD offset of the survey time series
CADENCE = {"2min": 2.0 / 1440.0, "30min": 1.0 / 48.0}
NPAR = {"quadratic": 2, "power-2": 2, "nonlinear": 4}
SIGMA = 5e-4               # white noise of the log-likelihood cases


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an optimiser or a notebook: one parameter vector, one transit, the default
        # precision, the numpy result of the reference's own call
        dict(name="rr_one_fp64", family="rr", precision="fp64", npv=1, npt=1000, nlc=1, npb=1, ns=1, times="window",
             law="quadratic", ecc=0.0, host=True),
        # an MCMC ensemble on one transit with an odd number of walkers and points
        dict(name="rr_chains_fp64", family="rr", precision="fp64", npv=77, npt=1501, nlc=1, npb=1, ns=1,
             times="window", law="quadratic", ecc=0.0, host=False),
        # a population over a space survey's sector: 2-min cadence over 27.4 d at BJD
        # scale, four passbands, the default precision
        dict(name="rr_survey_fp64", family="rr", precision="fp64", npv=8192, npt=19700, nlc=4, npb=4, ns=1,
             times="2min", law="quadratic", ecc=0.0, host=False),
        # long-cadence light curves of uneven lengths, supersampled, eccentric
        # orbits, the default precision
        dict(name="rr_cadence_fp64", family="rr", precision="fp64", npv=509, npt=60017, nlc=16, npb=4, ns=10,
             times="30min", law="power-2", ecc=0.3, host=False),
        # the sector population in split precision: the headline workload
        dict(name="rr_survey_split", family="rr", precision="split", npv=8192, npt=19700, nlc=4, npb=4, ns=1,
             times="2min", law="quadratic", ecc=0.0, host=False),
        # the long-cadence workload in split precision at its full population
        dict(name="rr_cadence_split", family="rr", precision="split", npv=4096, npt=118526, nlc=16, npb=4, ns=10,
             times="30min", law="power-2", ecc=0.3, host=False),
        # transmission spectroscopy over a sector: 200 channels, split precision
        dict(name="ts_survey_split", family="ts", precision="split", npv=64, npt=19700, npb=200, ns=1, times="2min",
             law="quadratic", ecc=0.0),
        # transmission spectroscopy of one observed transit, the default precision
        dict(name="ts_window_fp64", family="ts", precision="fp64", npv=100, npt=1203, npb=200, ns=5, times="window",
             law="quadratic", ecc=0.1),
        # secondary eclipses over a sector, the default precision
        dict(name="ecl_survey_fp64", family="ecl", precision="fp64", npv=1000, npt=19699, nlc=4, npb=0, ns=1,
             times="2min", ecc=0.1),
        # gradient-based sampling: log-likelihood forward and backward
        dict(name="lnl_grad_split", family="lnl", precision="split", npv=4096, npt=5000, ns=5, grad=True),
        # an ensemble sampler's step: a population held on the device to its
        # log-likelihoods, the default precision
        dict(name="lnl_lpf_fp64", family="lnl", precision="fp64", npv=1500, npt=2999, ns=1, grad=False),
        # a burst of mixed requests at a running server, results kept on the device
        dict(name="serve_burst", family="serve", nreq=24, npv=512, npt=20000),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["rr", "rr", "rr", "ts", "ecl", "lnl", "lnl", "serve"])
    precision = rng.choice(["fp64", "split"])
    if family == "rr":
        times = rng.choice(["window", "2min", "30min"])
        npt = _logint(rng, 200, 3000) if times == "window" else _logint(rng, 2000, 100000)
        most = (2.5e7 if precision == "fp64" else 2e8) / npt
        nlc = rng.choice([1, 2, 4, 9])
        return dict(family="rr", precision=precision, npv=max(1, min(_logint(rng, 1, 8192), int(most))), npt=npt,
                    nlc=nlc, npb=rng.choice([1, min(nlc, 2), min(nlc, 4)]), ns=rng.choice([1, 5, 10]), times=times,
                    law=rng.choice(["quadratic", "power-2", "nonlinear"]), ecc=rng.choice([0.0, 0.3]),
                    host=precision == "fp64" and rng.random() < 0.3)
    if family == "ts":
        times = rng.choice(["window", "2min"])
        npt = _logint(rng, 200, 3000) if times == "window" else _logint(rng, 2000, 20000)
        npb = _logint(rng, 10, 300)
        return dict(family="ts", precision=precision, npv=max(1, min(_logint(rng, 1, 256), int(1e8 / (npt * npb)))),
                    npt=npt, npb=npb, ns=rng.choice([1, 5, 10]), times=times,
                    law=rng.choice(["quadratic", "power-2", "nonlinear"]), ecc=rng.choice([0.0, 0.3]))
    if family == "ecl":
        times = rng.choice(["window", "2min"])
        npb = rng.choice([0, 0, _logint(rng, 2, 100)])      # 0: the eclipse model, else channels of the spectrum
        npt = _logint(rng, 200, 3000) if times == "window" else _logint(rng, 2000, 20000)
        most = 2e7 / (npt * max(1, npb))
        return dict(family="ecl", precision=precision, npv=max(1, min(_logint(rng, 1, 4096), int(most))), npt=npt,
                    nlc=1 if npb else rng.choice([1, 4]), npb=npb, ns=rng.choice([1, 5]), times=times,
                    ecc=rng.choice([0.0, 0.3]))
    if family == "lnl":
        npt = _logint(rng, 300, 8000)
        most = (4e6 if precision == "fp64" else 2e7) / npt
        return dict(family="lnl", precision=precision, npv=max(1, min(_logint(rng, 1, 4096), int(most))), npt=npt,
                    ns=rng.choice([1, 5]), grad=rng.random() < 0.5)
    return dict(family="serve", nreq=rng.randint(4, 32), npv=_logint(rng, 16, 512), npt=_logint(rng, 1000, 20000))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _ldc(rng, law, shape):
    """Limb-darkening coefficients [*shape, ncoef] over the ranges real stars have."""
    if law == "quadratic":
        return np.stack([rng.uniform(0.0, 0.6, shape), rng.uniform(0.0, 0.3, shape)], -1)
    if law == "power-2":
        return np.stack([rng.uniform(0.3, 0.9, shape), rng.uniform(0.3, 0.8, shape)], -1)
    return np.array([0.5, -0.2, 0.6, -0.25]) * rng.uniform(0.8, 1.2, shape + (4,))


def _orbits(rng, npv, ecc, pmin, pmax):
    a = rng.uniform(3.0, 20.0, npv)
    e = rng.uniform(0.0, ecc, npv) if ecc else np.zeros(npv)
    w = rng.uniform(0.0, 2.0 * np.pi, npv) if ecc else np.zeros(npv)
    return dict(p=rng.uniform(pmin, pmax, npv), a=a, i=np.arccos(rng.uniform(0.0, 0.9, npv) / a), e=e, w=w)


def _data(rng, c):
    """The observations (set_data's arguments) and the reference epoch."""
    npt, nlc, ns = c["npt"], c.get("nlc", 1), c["ns"]
    if c["times"] == "window":
        t_ref = 0.0
        step = 0.3 / npt
        time = -0.15 + 0.3 * (np.arange(npt) + rng.uniform(0.0, 1.0, npt)) / npt
        lcids = (np.arange(npt) * nlc) // npt
        exposure = step
    else:
        t_ref, step = T_BJD, CADENCE[c["times"]]
        exposure = step
        if c["times"] == "30min" and nlc > 1:       # light curves of uneven lengths over the same epoch
            wts = np.exp(rng.uniform(np.log(500.0), np.log(50000.0), nlc))
            n = np.maximum(1, np.floor(wts / wts.sum() * npt).astype(int))
            n[-1] += npt - n.sum()
            time = np.concatenate([t_ref + np.arange(m) * step for m in n])
            lcids = np.repeat(np.arange(nlc), n)
        else:
            time = t_ref + np.arange(npt) * step
            lcids = (np.arange(npt) * nlc) // npt
    data = dict(time=time, lcids=lcids.astype(np.int64), pbids=np.arange(nlc) % max(1, min(c.get("npb", 1), nlc)),
                nsamples=np.full(nlc, ns), exptimes=np.full(nlc, exposure if ns > 1 else 0.0))
    return data, t_ref


def _inputs(c, seed):
    """Everything a case computes from, as numpy arrays: observations and parameters."""
    rng = np.random.default_rng([seed, 17])
    f, npv = c["family"], c.get("npv")
    if f == "rr":
        data, t_ref = _data(rng, c)
        pmin = 1.0 if c["times"] == "window" else 0.5
        prm = dict(k=rng.uniform(0.05, 0.15, (npv, 1)), ldc=_ldc(rng, c["law"], (npv, c["npb"])),
                   t0=t_ref + rng.normal(0.0, 1e-3, (npv, 1)),
                   **_orbits(rng, npv, c["ecc"], pmin, 10.0 if c["times"] == "window" else 15.0))
        return data, prm
    if f == "ts":
        data, t_ref = _data(rng, dict(c, nlc=1, npb=1))
        mid = 0.0 if c["times"] == "window" else 13.7
        prm = dict(k=rng.uniform(0.09, 0.11, (npv, c["npb"])), ldc=_ldc(rng, c["law"], (npv, c["npb"])),
                   t0=t_ref + mid + rng.normal(0.0, 1e-3, npv), **_orbits(rng, npv, c["ecc"], 0.5, 15.0))
        return data, prm
    if f == "ecl":
        data, t_ref = _data(rng, dict(c, npb=1))
        orb = _orbits(rng, npv, c["ecc"], 1.0, 10.0)
        if c["times"] == "window":
            t0 = t_ref - _eclipse_shift(orb) + rng.normal(0.0, 1e-2, npv)    # the eclipse is in the window
        else:
            t0 = t_ref + rng.normal(0.0, 1e-3, npv)
        prm = dict(k=rng.uniform(0.05, 0.15, npv), t0=t0, rstar=1.0, **orb)
        if c["npb"]:
            prm["f"] = rng.uniform(1e-4, 3e-3, (npv, c["npb"]))
        return data, prm
    if f == "lnl":
        # a population around one planet's solution, as a sampler's chains sit
        npt = c["npt"]
        data = dict(time=np.linspace(-0.2, 0.2, npt), nsamples=[c["ns"]], exptimes=[1 / 48 if c["ns"] > 1 else 0.0])
        a, b, k = rng.uniform(4.0, 15.0), rng.uniform(0.0, 0.7), rng.uniform(0.06, 0.14)
        p, u = rng.uniform(2.0, 8.0), [rng.uniform(0.1, 0.5), rng.uniform(0.05, 0.25)]
        if c["grad"]:
            prm = dict(k=k * (1 + rng.normal(0, 0.02, (npv, 1))),
                       ldc=np.clip(np.array(u) + rng.normal(0, 0.02, (npv, 1, 2)), 0.01, None),
                       t0=rng.normal(0, 2e-4, (npv, 1)), p=p * (1 + rng.normal(0, 1e-4, npv)),
                       a=a * (1 + rng.normal(0, 0.01, npv)), i=np.arccos(b / a) + rng.normal(0, 1e-3, npv),
                       e=np.clip(0.1 + rng.normal(0, 0.01, npv), 0.01, None), w=1.0 + rng.normal(0, 0.05, npv))
        else:
            g, day = 6.6743e-11, 86400.0
            rho = a ** 3 * 3.0 * np.pi / (g * (p * day) ** 2) / 1e3
            pv = np.stack([rng.normal(0, 2e-4, npv), p * (1 + rng.normal(0, 1e-4, npv)),
                           rho * (1 + rng.normal(0, 0.03, npv)), np.clip(b + rng.normal(0, 0.02, npv), 0.0, None),
                           (k * (1 + rng.normal(0, 0.02, npv))) ** 2, rng.uniform(0.2, 0.6, npv),
                           rng.uniform(0.2, 0.6, npv)], -1)
            prm = dict(pv=pv)
        half = (1 + k) / (2 * np.pi * a / p)
        obs = 1.0 - k ** 2 * (np.abs(data["time"]) < half) + rng.normal(0, SIGMA, npt)
        return dict(data, obs=obs), prm
    reqs = []
    mix = np.random.default_rng([c["nreq"], npv, c["npt"]])      # the requests' sizes belong to the case
    for _ in range(c["nreq"]):
        kind = "ts" if mix.uniform() < 0.2 else "rr"
        law = ["quadratic", "power-2", "nonlinear"][int(mix.integers(0, 3))]
        n = int(np.exp(mix.uniform(0.0, np.log(npv))))
        n, npb = (max(1, n // 16), 200) if kind == "ts" else (n, 1)
        npt = int(np.exp(mix.uniform(np.log(500.0), np.log(c["npt"]))))
        ns = int(mix.choice([1, 5, 10]))
        data = dict(time=T_BJD + np.arange(npt) * CADENCE["2min"], nsamples=[ns],
                    exptimes=[CADENCE["2min"] if ns > 1 else 0.0])
        prm = dict(k=rng.uniform(0.09, 0.11, (n, npb)) if kind == "ts" else rng.uniform(0.05, 0.15, (n, 1)),
                   ldc=_ldc(rng, law, (n, npb)), t0=T_BJD + rng.normal(0.0, 1e-3, n),
                   **_orbits(rng, n, 0.0, 0.5, 15.0))
        reqs.append((kind, law, data, prm))
    return reqs, None


_server = None


def _the_server():
    """The one server that a serving program keeps for its life."""
    global _server
    if _server is None:
        from pytransit_gb300.serving import RRServer
        _server = RRServer(hbm_budget=16e9, result="device")
    return _server


def prepare(case, seed):
    c = dict(case)
    f = c["family"]
    data, prm = _inputs(c, seed)
    if f == "serve":
        return dict(c=c, server=_the_server(), reqs=data)
    dev = torch.device("cuda", torch.cuda.current_device())
    if f == "ecl":
        from pytransit_gb300 import EclipseModel, EclipseSpectroscopyModel
        m = (EclipseSpectroscopyModel if c["npb"] else EclipseModel)(precision=c["precision"])
        m.set_data(**data)
        return dict(c=c, m=m, prm=prm)
    from pytransit_gb300 import RoadRunnerModel, TransmissionSpectroscopyModel
    if f == "ts":
        m = TransmissionSpectroscopyModel(c["law"], precision=c["precision"])
        m.set_data(**data)
        return dict(c=c, m=m, prm=prm)
    if f == "rr":
        m = RoadRunnerModel(c["law"], precision=c["precision"])
        m.set_data(**data)
        return dict(c=c, m=m, prm=prm)
    m = RoadRunnerModel("quadratic", precision=c["precision"])
    obs = torch.as_tensor(data.pop("obs")).to(dev)
    m.set_data(**data)
    tens = {n: torch.as_tensor(v).to(dev).requires_grad_(c["grad"]) for n, v in prm.items()}
    return dict(c=c, m=m, obs=obs, prm=tens)


_ORDER = ("k", "ldc", "t0", "p", "a", "i", "e", "w")
_GRAD = ("k", "t0", "p", "a", "i", "e", "w", "ldc")


def run(state):
    c = state["c"]
    f = c["family"]
    if f == "serve":
        futures = [state["server"].submit(*r) for r in state["reqs"]]
        return [q.result() for q in futures]
    m, prm = state["m"], state["prm"]
    if f == "rr":
        return m.evaluate(*(prm[n] for n in _ORDER), copy=c["host"])
    if f == "ts":
        return m.evaluate(*(prm[n] for n in _ORDER), copy=False)
    if f == "ecl":
        lead = (prm["f"],) if c["npb"] else ()
        return m.evaluate(*lead, *(prm[n] for n in ("k", "t0", "p", "a", "i", "e", "w", "rstar")), copy=False)
    if c["grad"]:
        from pytransit_gb300.lnlike import LogLikelihood
        x = [prm[n] for n in _GRAD]
        lnl = LogLikelihood.apply(m, state["obs"], SIGMA, *x)
        return dict(lnl=lnl.detach(), grad=torch.autograd.grad(lnl.sum(), x))
    from pytransit_gb300 import lpf
    return lpf.lnlikelihood(m, state["obs"], SIGMA, prm["pv"], 0.0)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _rr_work(npv, npt, ns, npb_out, nbytes, npar_values, frac):
    """Inputs once, outputs once; per point a phase fold and a box test (12
    operations), per in-transit sample the separation, the LD lerp and the
    overlap area (80 operations), per further channel 6 operations a point."""
    out = nbytes * npv * npt * npb_out
    flops = npv * npt * (12.0 + frac * ns * 80.0) + 6.0 * frac * npv * npt * (npb_out - 1)
    return dict(bytes=float(out + 12 * npt + 8 * npar_values), flops=float(flops))


def work(case):
    c = case
    f = c["family"]
    frac = {"window": 0.5, "2min": 0.04, "30min": 0.05}.get(c.get("times"), 0.5)
    if f == "serve":
        # the expectation over the requests' distribution
        lg = math.log(c["npv"])
        mean_npv, mean_npt = (c["npv"] - 1) / lg, (c["npt"] - 500) / math.log(c["npt"] / 500.0)
        rr = _rr_work(mean_npv, mean_npt, 5.3, 1, 4, 9 * mean_npv, 0.04)
        ts = _rr_work(max(1.0, mean_npv / 16), mean_npt, 5.3, 200, 4, 600 * max(1.0, mean_npv / 16), 0.04)
        return {q: c["nreq"] * (0.8 * rr[q] + 0.2 * ts[q]) for q in ("bytes", "flops")}
    npv, npt, ns = c["npv"], c["npt"], c["ns"]
    size = 8 if c["precision"] == "fp64" else 4
    if f == "rr":
        return _rr_work(npv, npt, ns, 1, size, npv * (7 + c["npb"] * NPAR[c["law"]]), frac)
    if f == "ts":
        return _rr_work(npv, npt, ns, c["npb"], size, npv * (6 + c["npb"] * (1 + NPAR[c["law"]])), frac)
    if f == "ecl":
        return _rr_work(npv, npt, ns, max(1, c["npb"]), size, npv * (8 + c["npb"]), frac)
    ncol = 9
    flops = npv * npt * (12.0 + 0.5 * ns * (80.0 + (25.0 * ncol if c["grad"] else 0.0)))
    return dict(bytes=float(16 * npt + 8 * npv * (ncol + 1 + (ncol if c["grad"] else 0))), flops=flops)


# ---------------------------------------------------------------------------
# The same values in plain torch, 64 bits
# ---------------------------------------------------------------------------
NK, NG, KMIN, KMAX = 256, 100, 0.005, 0.5
DK, DG = (KMAX - KMIN) / NK, (1.0 - 1e-7) / (NG - 1)


def _dev():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _t(x):
    return torch.as_tensor(np.asarray(x, dtype=np.float64), device=_dev())


def _zgrid():
    """Radial grid: 20 bins uniform in z up to 0.7, 20 uniform in mu to the limb."""
    nin, nedge, zcut = 20, 20, 0.7
    ze, zm = np.zeros(nin + nedge), np.zeros(nin + nedge)
    ze[:nin - 1] = (np.arange(nin - 1) + 1) * (zcut / nin)
    dmu = math.sqrt(1.0 - zcut ** 2) / nedge
    for i in range(nedge + 1):
        ze[-i - 1] = math.sqrt(1.0 - (i * dmu) ** 2)
    zm[1:] = 0.5 * (ze[:-1] + ze[1:])
    return ze, np.sqrt(1.0 - zm ** 2)


def _lens_acos(r1, r2, b):
    """Overlap area of two circles, the two-arccosine form of the weight tables."""
    r1, r2, b = torch.broadcast_tensors(r1, r2, b)
    bs = torch.where(b > 0, b, torch.ones_like(b))
    x = ((b * b + r2 * r2 - r1 * r1) / (2 * bs * r2)).clamp(-1.0, 1.0)
    y = ((b * b + r1 * r1 - r2 * r2) / (2 * bs * r1)).clamp(-1.0, 1.0)
    q = ((-b + r2 + r1) * (b + r2 - r1) * (b - r2 + r1) * (b + r2 + r1)).clamp(min=0.0)
    area = r2 * r2 * torch.acos(x) + r1 * r1 * torch.acos(y) - 0.5 * torch.sqrt(q)
    area = torch.where(b - r2 <= -r1, math.pi * r1 * r1, area)
    area = torch.where(r1 >= b + r2, math.pi * r2 * r2, area)
    return torch.where(r1 < b - r2, torch.zeros_like(area), area)


def _weights(k):
    """Normalised ring weights [*k.shape, NG, nz] of a planet of radius k."""
    ze = _t(_zgrid()[0])
    g = _t(np.linspace(0.0, 1.0 - 1e-7, NG))
    kk = k[..., None, None]
    area = _lens_acos(ze, kk, g[:, None] * (1.0 + kk))
    wts = torch.diff(area, dim=-1, prepend=torch.zeros_like(area[..., :1]))
    return wts / wts.sum(-1, keepdim=True)


def _profile(law, ldc, mu):
    """The LD profile [..., nmu] of coefficients [..., ncoef]."""
    u = [ldc[..., j:j + 1] for j in range(ldc.shape[-1])]
    m = 1.0 - mu
    if law == "quadratic":
        return 1.0 - u[0] * m - u[1] * m * m
    if law == "power-2":
        return 1.0 - u[0] * (1.0 - mu ** u[1])
    return 1.0 - u[0] * (1.0 - mu.sqrt()) - u[1] * m - u[2] * (1.0 - mu ** 1.5) - u[3] * (1.0 - mu * mu)


def _integral(law, ldc):
    """The disk integral, analytic or by the 200-point trapezoid."""
    if law == "quadratic":
        return 2.0 * math.pi / 12.0 * (-2.0 * ldc[..., 0] - ldc[..., 1] + 6.0)
    if law == "power-2":
        c, al = ldc[..., 0], ldc[..., 1]
        return 2.0 * math.pi * (-c * al + al + 2.0) / (2.0 * al + 4.0)
    mu = _t(np.linspace(1.0, 0.0, 200))
    z = torch.sqrt(1.0 - mu * mu)
    return 2.0 * math.pi * torch.trapezoid(z * _profile(law, ldc, mu), z, dim=-1)


def _orbit(p, a, i, e, w, s=1.0):
    """Taylor coefficients of the sky position about the transit (s = 1) or the
    eclipse (s = -1): two lists of five."""
    n, se = 2.0 * math.pi / p, torch.sqrt(1.0 - e * e)
    sf, cf = s * torch.cos(w), s * torch.sin(w)
    r = a * (1.0 - e * e) / (1.0 + e * cf)
    x = [torch.zeros_like(r), -s * n * a * (1.0 + e * cf) / se]
    y = [s * r, s * n * a * e * sf / se]
    mu = n * n * a ** 3
    q = [y[0] * y[0], 2.0 * y[0] * y[1]]
    h = [1.0 / (q[0] * torch.sqrt(q[0]))]
    for v in (x, y):
        v.append(-mu * h[0] * v[0] / 2.0)
    h.append(-1.5 * q[1] * h[0] / q[0])
    for v in (x, y):
        v.append(-mu * (h[0] * v[1] + h[1] * v[0]) / 6.0)
    q.append(2.0 * (x[0] * x[2] + y[0] * y[2]) + x[1] * x[1] + y[1] * y[1])
    h.append((-2.5 * q[1] * h[1] - 3.0 * q[2] * h[0]) / (2.0 * q[0]))
    for v in (x, y):
        v.append(-mu * (h[0] * v[2] + h[1] * v[1] + h[2] * v[0]) / 12.0)
    ci = torch.cos(i)
    return [-v for v in x], [-ci * v for v in y]


def _sep(t, xs, ys):
    x, y = xs[4], ys[4]
    for j in (3, 2, 1, 0):
        x, y = xs[j] + t * x, ys[j] + t * y
    return torch.sqrt(x * x + y * y)


def _contact(k, xs, ys, sign):
    """The outer contact before (-1) or after (1) conjunction, by bisection."""
    lo, hi = torch.zeros_like(k), sign * 2.0 / xs[1].abs()
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        inside = _sep(mid, xs, ys) < 1.0 + k
        lo, hi = torch.where(inside, mid, lo), torch.where(inside, hi, mid)
    return 0.5 * (lo + hi)


def _area(k, z):
    """Overlap area of the unit disk and a planet of radius k < 1, and kappa_0."""
    inner, limb = z <= 1.0 - k, (z > 1.0 - k) & (z < 1.0 + k)
    zs = torch.where(limb, z, torch.ones_like(z))
    kite = 0.5 * torch.sqrt((zs + (1.0 + k)) * (k - (zs - 1.0)) * (k + (zs - 1.0)) * (zs + (1.0 - k)))
    k0 = torch.atan2(2.0 * kite, (k - 1.0) * (k + 1.0) + zs * zs)
    k1 = torch.atan2(2.0 * kite, (1.0 - k) * (1.0 + k) + zs * zs)
    zero = torch.zeros_like(z)
    area = torch.where(inner, math.pi * k * k + zero, torch.where(limb, k1 + k * k * k0 - kite, zero))
    return area, torch.where(inner, math.pi + zero, torch.where(limb, k0, zero))


def _fold(t, t0, p):
    epoch = torch.floor((t - t0 + 0.5 * p) / p)
    return t - (t0 + epoch * p)


def _samples(ns, ex):
    for s in range(ns):
        yield ex * ((s + 0.5) / ns - 0.5)


def _lerp_at(z, k):
    g = z / (1.0 + k)
    j = torch.floor(g.detach() / DG).clamp(0, NG - 2).long()
    return j, (g - j * DG) / DG


def _rr_means(law, k, ldc, table):
    """LD means [npv, npb, NG] at the k-interpolated weight table."""
    mu = _t(_zgrid()[1])
    ik = torch.floor((k.detach() - KMIN) / DK).long()
    ak = ((k - KMIN - ik * DK) / DK)[:, None, None]
    prof = _profile(law, ldc, mu)
    return ((1.0 - ak) * torch.einsum("pgz,pbz->pbg", table[ik], prof) +
            ak * torch.einsum("pgz,pbz->pbg", table[ik + 1], prof))


def _rr_deficit(ii, tc, ns, ex, k, xs, ys, means, pb, istar):
    """The deficit of points (ii: their parameter vector, tc: their time from conjunction)."""
    xs, ys, kk = [v[ii] for v in xs], [v[ii] for v in ys], k[ii]
    d = torch.zeros_like(tc)
    for off in _samples(ns, ex):
        z = _sep(tc + off, xs, ys)
        j, fr = _lerp_at(torch.minimum(z, 1.0 + kk), kk)
        mean = (1.0 - fr) * means[ii, pb, j] + fr * means[ii, pb, j + 1]
        d = d + torch.where(z < 1.0 + kk, mean * _area(kk, z)[0], torch.zeros_like(z))
    return d / (ns * istar[ii, pb])


def _exact_rr(law, data, prm):
    dev = _dev()
    time = _t(data["time"])
    lc = torch.as_tensor(data.get("lcids", np.zeros(time.numel(), np.int64)), device=dev)
    pbs = torch.as_tensor(data.get("pbids", np.zeros(1, np.int64)), device=dev)
    ns, ex = int(data["nsamples"][0]), float(data["exptimes"][0])
    k, t0 = _t(prm["k"])[:, 0], _t(prm["t0"]).reshape(-1)
    ldc, p = _t(prm["ldc"]), _t(prm["p"])
    xs, ys = _orbit(p, *(_t(prm[n]) for n in ("a", "i", "e", "w")))
    t1, t4 = (_contact(k, xs, ys, s) for s in (-1.0, 1.0))
    kgrid = _t(KMIN + np.arange(NK) * ((KMAX - KMIN) / (NK - 1)))
    table = _weights(kgrid)
    out = torch.ones((k.numel(), time.numel()), dtype=torch.float64, device=dev)
    istar = _integral(law, ldc)
    pad = 0.003 + ex
    step = max(1, int(3e7) // time.numel())
    for q in range(0, k.numel(), step):
        sl = slice(q, q + step)
        tc = _fold(time, t0[sl, None], p[sl, None])
        ii, jj = torch.nonzero((tc >= (t1[sl] - pad)[:, None]) & (tc <= (t4[sl] + pad)[:, None]), as_tuple=True)
        d = _rr_deficit(ii, tc[ii, jj], ns, ex, k[sl], [v[sl] for v in xs], [v[sl] for v in ys],
                        _rr_means(law, k[sl], ldc[sl], table), pbs[lc[jj]], istar[sl])
        out[q + ii, jj] = 1.0 - d
    return out


def _exact_ts(law, data, prm):
    time, kb, ldc, p = _t(data["time"]), _t(prm["k"]), _t(prm["ldc"]), _t(prm["p"])
    ns, ex = int(data["nsamples"][0]), float(data["exptimes"][0])
    km, kx = kb.mean(1), kb.max(1).values
    xs, ys = _orbit(p, *(_t(prm[n]) for n in ("a", "i", "e", "w")))
    t1, t4 = (_contact(km, xs, ys, s) for s in (-1.0, 1.0))
    means = torch.einsum("pgz,pbz->pbg", _weights(km), _profile(law, ldc, _t(_zgrid()[1])))
    istar, pad = _integral(law, ldc), 0.0015 + ex
    tc = _fold(time, _t(prm["t0"]).reshape(-1, 1), p[:, None])
    out = torch.ones(kb.shape + (time.numel(),), dtype=torch.float64, device=kb.device)
    for q in range(kb.shape[0]):
        jj = torch.nonzero((tc[q] >= t1[q] - pad) & (tc[q] <= t4[q] + pad))[:, 0]
        d = torch.zeros((kb.shape[1], jj.numel()), dtype=torch.float64, device=kb.device)
        for off in _samples(ns, ex):
            z = _sep(tc[q, jj] + off, [v[q] for v in xs], [v[q] for v in ys])
            area, kappa = _area(km[q], z)
            j, fr = _lerp_at(torch.minimum(z, 1.0 + km[q]), km[q])
            mean = (1.0 - fr) * means[q][:, j] + fr * means[q][:, j + 1]
            full = (kb[q] ** 2 / km[q] ** 2)[:, None] * area
            part = area + (kb[q] - km[q])[:, None] * (2.0 * km[q] * kappa)
            occ = torch.where(z <= 1.0 - kx[q], full, part)
            d = d + torch.where(z < 1.0 + km[q], mean * occ, torch.zeros_like(mean))
        out[q][:, jj] = 1.0 - d / (ns * istar[q][:, None])
    return out


def _eclipse_shift(orb):
    """Days from mid-transit to mid-eclipse."""
    p, e, w = orb["p"], orb["e"], orb["w"]
    se = np.sqrt(1.0 - e * e)
    m = []
    for f in (0.5 * np.pi - w, 0.5 * np.pi + np.pi - w):
        ea = np.arctan2(se * np.sin(f), e + np.cos(f))
        m.append(ea - e * np.sin(ea))
    s = (m[1] - m[0]) * p / (2.0 * np.pi)
    return np.where(s > 0.0, s, p + s)


def _exact_ecl(data, prm):
    time, k, p = _t(data["time"]), _t(prm["k"]), _t(prm["p"])
    a, i, e, w = (_t(prm[n]) for n in ("a", "i", "e", "w"))
    ns, ex = int(data["nsamples"][0]), float(data["exptimes"][0])
    f = _t(prm["f"]) if "f" in prm else None
    r = [a * (1.0 - e * e) / (1.0 + e * torch.cos(u - w)) for u in (0.5 * math.pi, 1.5 * math.pi)]
    ltt = (r[0] + r[1]) * torch.sin(i) * prm["rstar"] * 6.957e8 / 299792458.0 / 86400.0
    te = _t(prm["t0"]) + _t(_eclipse_shift(prm)) + ltt
    xs, ys = _orbit(p, a, i, e, w, -1.0)
    t1, t4 = (_contact(k, xs, ys, s) for s in (-1.0, 1.0))
    pad = (0.003 if f is None else 0.0015) + ex
    shape = (k.numel(), time.numel()) if f is None else tuple(f.shape) + (time.numel(),)
    out = torch.ones(shape, dtype=torch.float64, device=k.device)
    if f is None:
        out *= (math.pi * k * k)[:, None]
    tc = _fold(time, te[:, None], p[:, None])
    ii, jj = torch.nonzero((tc >= (t1 - pad)[:, None]) & (tc <= (t4 + pad)[:, None]), as_tuple=True)
    kk, area = k[ii], torch.zeros(ii.numel(), dtype=torch.float64, device=k.device)
    for off in _samples(ns, ex):
        area = area + _area(kk, _sep(tc[ii, jj] + off, [v[ii] for v in xs], [v[ii] for v in ys]))[0] / ns
    if f is None:
        out[ii, jj] = math.pi * kk * kk - area
    else:
        ff = f[ii]
        out[ii, :, jj] = 1.0 - ff * (area / math.pi)[:, None] / (1.0 + ff * (kk * kk)[:, None])
    return out


def _exact_lnl(c, data, prm):
    time, dobs = _t(data["time"]), _t(data["obs"]) - 1.0
    ns, ex = int(data["nsamples"][0]), float(data["exptimes"][0])
    if c["grad"]:
        x = {n: _t(prm[n]) for n in _GRAD}
    else:
        pv = _t(prm["pv"])
        a = (6.6743e-11 / (3.0 * math.pi)) ** (1.0 / 3.0) * ((pv[:, 1] * 86400.0) ** 2 * 1e3 * pv[:, 2]) ** (1.0 / 3.0)
        s, v = torch.sqrt(pv[:, 5]), 2.0 * pv[:, 6]
        zero = torch.zeros_like(a)
        x = dict(k=torch.sqrt(pv[:, 4:5]), t0=pv[:, 0:1], p=pv[:, 1], a=a, i=torch.acos(pv[:, 3] / a), e=zero, w=zero,
                 ldc=torch.stack([s * v, s * (1.0 - v)], -1)[:, None, :])
    table = _weights(_t(KMIN + np.arange(NK) * ((KMAX - KMIN) / (NK - 1))))
    npv = x["p"].numel()
    const = -time.numel() * (math.log(SIGMA) + 0.5 * math.log(2.0 * math.pi))
    const = const - 0.5 * float((dobs * dobs).sum()) / SIGMA ** 2
    lnl = torch.empty(npv, dtype=torch.float64, device=time.device)
    grads = {n: torch.empty_like(v) for n, v in x.items()}
    step = max(1, int(4e6) // time.numel())
    for q in range(0, npv, step):
        y = {n: v[q:q + step].clone().requires_grad_(c["grad"]) for n, v in x.items()}
        k, t0, p = y["k"][:, 0], y["t0"][:, 0], y["p"]
        xs, ys = _orbit(p, y["a"], y["i"], y["e"], y["w"])
        with torch.no_grad():
            t1, t4 = (_contact(k, xs, ys, s) for s in (-1.0, 1.0))
            tc = _fold(time, t0[:, None], p[:, None])
            epoch = torch.round((time - t0[:, None] - tc) / p[:, None])
            pad = 0.003 + ex
            ii, jj = torch.nonzero((tc >= (t1 - pad)[:, None]) & (tc <= (t4 + pad)[:, None]), as_tuple=True)
        tb = time[jj] - (t0[ii] + epoch[ii, jj] * p[ii])
        d = _rr_deficit(ii, tb, ns, ex, k, xs, ys, _rr_means("quadratic", k, y["ldc"], table),
                        torch.zeros_like(ii), _integral("quadratic", y["ldc"]))
        terms = -(dobs[jj] + 0.5 * d) * d / SIGMA ** 2
        part = torch.zeros_like(p).index_add(0, ii, terms)
        lnl[q:q + step] = part.detach() + const
        if c["grad"]:
            for n, gq in zip(y, torch.autograd.grad(part.sum(), list(y.values()))):
                grads[n][q:q + step] = gq
    return dict(lnl=lnl, grad=tuple(grads[n] for n in _GRAD)) if c["grad"] else lnl


def exact(case, seed):
    c = dict(case)
    data, prm = _inputs(c, seed)
    f = c["family"]
    if f == "rr":
        out = _exact_rr(c["law"], data, prm).squeeze()
    elif f == "ts":
        out = _exact_ts(c["law"], data, prm)
    elif f == "ecl":
        out = _exact_ecl(data, prm)
    elif f == "lnl":
        out = _exact_lnl(c, data, prm)
    else:
        out = [(_exact_rr if kind == "rr" else _exact_ts)(law, d, q) for kind, law, d, q in data]
    return out
