"""The FP64 log-likelihood's gradient against torch's automatic differentiation
of the same discretised model (the oracle's weight tables, the kite area, the
orbit's Taylor coefficients) in FP64 on the host.

Tolerance: 1e-9 of each column's largest value.  The kernel's operations are
within a few ulps, the largest amplification is the k derivative's table
difference over dk (1e-15 / 2e-3), and sums of up to 1e4 terms.  For a k outside
the table the mean's derivative is defined as the central difference of the 2D
table at k (1 +- 1e-6), which carries the tables' 1e-15 as 1e-9: 1e-8 there.
"""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def area(k, z):
    """Overlap of the unit disk and a disk of radius k, differentiable (k, z broadcast)."""
    limb = ((1.0 - k).abs() < z) & (z < 1.0 + k)
    zs, ks = torch.where(limb, z, torch.ones_like(z)), torch.where(limb, k, 0.5 * torch.ones_like(k))
    s1, s0 = (1.0 + ks) ** 2 - zs ** 2, zs ** 2 - (1.0 - ks) ** 2
    kite = 0.5 * torch.sqrt(s1 * s0)
    a = (torch.atan2(2.0 * kite, 1.0 - ks ** 2 + zs ** 2) + ks ** 2 * torch.atan2(2.0 * kite, ks ** 2 - 1.0 + zs ** 2) -
         kite)
    small = torch.minimum(k, torch.ones_like(k))
    full = torch.where(z <= (1.0 - k).abs(), np.pi * small ** 2 * torch.ones_like(z), torch.zeros_like(z))
    return torch.where(limb, a, full)


def orbit(p, a, i, e, w):
    """Coefficients of x(t), y(t): the series of r'' = -mu r / |r|^3 from mid-transit."""
    n, se = 2 * np.pi / p, torch.sqrt(1 - e * e)
    r = a * (1 - e * e) / (1 + e * torch.sin(w))
    x, y = [torch.zeros_like(r), -n * a * (1 + e * torch.sin(w)) / se], [r, n * a * e * torch.cos(w) / se]
    mu = n * n * a ** 3
    s = []          # series of |r|^-3
    for m in range(3):
        q = [sum(v[j] * v[l - j] for v in (x, y) for j in range(l + 1)) for l in range(m + 1)]   # of |r|^2
        s.append(q[0] ** -1.5 if m == 0 else
                 sum((-1.5 * j - (m - j)) * q[j] * s[m - j] for j in range(1, m + 1)) / (m * q[0]))
        for v in (x, y):
            v.append(-mu * sum(s[j] * v[m - j] for j in range(m + 1)) / ((m + 1) * (m + 2)))
    return [-v for v in x], [-torch.cos(i) * v for v in y]


def model_lnl(ref, data, obs, sigma, k, t0, p, a, i, e, w, ldc):
    """lnL[npv], differentiable in the parameters (k[npv, nkc], t0[npv, nep], ldc[npv, npb, 2])."""
    npv, npb = p.numel(), ldc.shape[1]
    time, lcids = data['time'], np.asarray(data['lcids'])
    mu = torch.as_tensor(ref.mu)
    xs, ys = orbit(p, a, i, e, w)
    out = []
    for q in range(npv):
        prof = 1 - ldc[q, :, :1] * (1 - mu) - ldc[q, :, 1:] * (1 - mu) ** 2
        istar = 2 * np.pi / 12 * (6 - 2 * ldc[q, :, 0] - ldc[q, :, 1])
        k0 = float(k[q, 0].detach())
        if ref.klims[0] <= k0 <= ref.klims[1] - ref.dk:
            ik = int(np.floor((k0 - ref.klims[0]) / ref.dk))
            ak = (k[q, 0] - ref.klims[0] - ik * ref.dk) / ref.dk
            W0, W1 = (torch.as_tensor(ref.weights[j]) for j in (ik, ik + 1))
            means = (1 - ak) * (prof @ W0.T) + ak * (prof @ W1.T)
        else:
            h = 1e-6 * max(k0, 1e-3)
            W, Wp, Wm = (torch.as_tensor(oracle.weights_2d(v, ref.ze, ref.ng)[1]) for v in (k0, k0 + h, k0 - h))
            means = prof @ W.T + (k[q, 0] - k0) * (prof.detach() @ ((Wp - Wm) / (2 * h)).T)
        c = np.array([float(v[q].detach()) for v in xs + ys])
        t1, t4 = oracle.bounding_box(k0, c)
        lnl = 0.0
        for lc in range(len(data['pbids'])):
            pb, ep, ns, ex = data['pbids'][lc], data['epids'][lc], data['nsamples'][lc], data['exptimes'][lc]
            sel = lcids == lc
            t, tq, pq = time[sel], float(t0[q, ep].detach()), float(p[q].detach())
            epoch = np.floor((t - tq + 0.5 * pq) / pq)
            tc = t - (tq + epoch * pq)
            box = (t1 - (0.003 + ex) <= tc) & (tc <= t4 + (0.003 + ex))
            o = torch.as_tensor(obs[sel]) - 1
            lnl = lnl - t.size * (np.log(sigma[lc]) + 0.5 * np.log(2 * np.pi)) - 0.5 * (o * o).sum() / sigma[lc] ** 2
            # the rounded fold, moved by the parameters' derivatives
            tb = (torch.as_tensor(tc[box]) - (t0[q, ep] - tq) - torch.as_tensor(epoch[box]) * (p[q] - pq))
            kk = k[q, pb if k.shape[1] > 1 else 0]
            d = torch.zeros_like(tb)
            for s in range(ns):
                ts = tb + ex * ((s + 0.5) / ns - 0.5)
                x = sum(xs[m][q] * ts ** m for m in range(5))
                y = sum(ys[m][q] * ts ** m for m in range(5))
                z = torch.sqrt(x * x + y * y)
                g = z / (1 + kk)
                j = torch.clamp(torch.floor(g.detach() / ref.dg), 0, ref.ng - 2).long()
                fr = (g - j.double() * ref.dg) / ref.dg
                mean = (1 - fr) * means[pb][j] + fr * means[pb][j + 1]
                d = d + torch.where(z < 1 + kk, mean * area(kk, z), torch.zeros_like(z))
            d = d / (ns * istar[pb])
            lnl = lnl - ((o[torch.as_tensor(box)] + 0.5 * d) * d).sum() / sigma[lc] ** 2
        out.append(lnl)
    return torch.stack(out)


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("k0,npb,nep,start,period,tol", [
    (0.05, 1, 1, 0.0, 3.0, 1e-9), (0.12, 3, 2, 0.0, 3.0, 1e-9),
    (0.1, 1, 1, 2459000.0, 0.8, 1e-9),              # three to six million epochs from t0
    (0.1, 1, 1, 2459000.0, 0.38, 1e-9), (0.1, 1, 1, 2459000.0, 0.45, 1e-9), (0.1, 1, 1, 2459000.0, 0.51, 1e-9),
    (0.1, 2, 1, 2459000.0, 11.0, 1e-9),
    (0.7, 1, 1, 0.0, 3.0, 1e-8), (1.2, 2, 1, 0.0, 3.0, 1e-8)])
def test_gradient_against_autograd(k0, npb, nep, start, period, tol, ns):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(int(period * 10) + npb + ns)
    npv, per = 4, 700
    first = np.ceil(start / period) * period
    time = np.concatenate([first + 3 * j * period + np.linspace(-0.12, 0.11, per) for j in range(npb)])
    data = dict(time=time, lcids=np.repeat(np.arange(npb), per), pbids=np.arange(npb), nsamples=[ns] * npb,
                exptimes=[0.02 if ns > 1 else 0.0] * npb, epids=np.arange(npb) % nep)
    a = rng.uniform(6, 12, npv) * (period / 3.0) ** (2 / 3)
    spread = 1e-4 / max(1.0, start / period)
    prm = dict(k=k0 * rng.uniform(0.9, 1.1, (npv, npb)), t0=rng.normal(0, 1e-3, (npv, nep)),
               p=period + rng.normal(0, spread, npv), a=a, i=np.arccos(rng.uniform(0.1, 0.8, npv) / a),
               e=rng.uniform(0.05, 0.2, npv), w=rng.uniform(0, 6, npv), ldc=rng.uniform(0.1, 0.4, (npv, npb, 2)))
    sigma = rng.uniform(0.8e-3, 1.2e-3, npb)
    obs = 1.0 - 0.8 * k0 ** 2 * (np.abs((time - first + 1.5 * period) % period - 0.5 * period) < 0.05)
    obs = obs + rng.normal(0, 1e-3, time.size)
    ref = oracle.OracleRoadRunner('quadratic')
    x = {n: torch.as_tensor(v).requires_grad_(True) for n, v in prm.items()}
    want = model_lnl(ref, data, obs, sigma, *(x[n] for n in ('k', 't0', 'p', 'a', 'i', 'e', 'w', 'ldc')))
    gw = torch.autograd.grad(want.sum(), list(x.values()))
    gw = np.concatenate([v.reshape(npv, -1).numpy() for v in gw], 1)
    m = RoadRunnerModel('quadratic')
    m.set_data(**data)
    lnl, g = lnlikelihood(m, obs, sigma, *(prm[n] for n in ('k', 'ldc', 't0', 'p', 'a', 'i', 'e', 'w')), grad=True)
    np.testing.assert_allclose(lnl, want.detach().numpy(), rtol=1e-10)
    assert (np.abs(gw).max(0) > 0).all()
    err = np.abs(g - gw).max(0) / np.abs(gw).max(0)
    assert (err <= tol).all(), err
