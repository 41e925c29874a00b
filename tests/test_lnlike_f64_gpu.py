"""The FP64 log-likelihood and its adjoint at the sizes where the kernel
changes form: tiles of many light curves, more light curves than are staged,
more samples than a queue chunk holds, one point, several epochs and passbands,
radius ratios on both sides of the kite form's range.

lnL: 1e-9 relative against the oracle's flux (the FP64 path's tolerance; the
sum's own rounding is far below).  Gradient: against the split path's kernel,
which shares none of the FP64 kernel's sample arithmetic, to 1e-4 of each
column's largest value (the split path's tolerance).  (Difference quotients of
the oracle's lnL do not resolve these cases: with 78,000 samples some cross a
kink of the piecewise-linear LD tables at any step above the times' rounding.)
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1, 1, 0.1), (1, 400, 1, 1, 0.1), (1, 260, 300, 1, 0.1), (3, 129, 5, 2, 0.1), (40, 9, 2, 3, 0.15),
         (2, 200, 1, 1, 1.2), (2, 300, 3, 2, 0.6)]


def problem(nlc, per, ns, npb, k0):
    rng = np.random.default_rng(nlc * per + ns)
    npv = 5
    npb = min(npb, nlc)
    time = np.concatenate([3.0 * j + (np.linspace(-0.12, 0.11, per) if per > 1 else np.array([0.01])) for j in range(nlc)])
    data = dict(time=time, lcids=np.repeat(np.arange(nlc), per), pbids=np.arange(nlc) % npb,
                nsamples=[ns] * nlc, exptimes=[0.02 if ns > 1 else 0.0] * nlc, epids=np.arange(nlc) % 2)
    a = rng.uniform(6, 12, npv)
    prm = dict(k=k0 * rng.uniform(0.9, 1.1, (npv, npb)), ldc=rng.uniform(0.1, 0.4, (npv, npb, 2)),
               t0=rng.normal(0, 1e-3, (npv, 2 if nlc > 1 else 1)), p=3.0 + rng.normal(0, 1e-3, npv), a=a,
               i=np.arccos(rng.uniform(0.1, 0.8, npv) / a), e=rng.uniform(0.05, 0.2, npv), w=rng.uniform(0, 6, npv))
    obs = 1.0 - 0.8 * k0 ** 2 * (np.abs((time + 1.5) % 3.0 - 1.5) < 0.05) + rng.normal(0, 1e-3, time.size)
    return data, prm, obs, rng.uniform(0.8e-3, 1.2e-3, nlc)


def oracle_lnl(ref, data, prm, obs, sigma):
    f = ref.evaluate(*(prm[n] for n in ('k', 'ldc', 't0', 'p', 'a', 'i', 'e', 'w'))).reshape(prm['p'].size, -1)
    s = sigma[data['lcids']]
    return (-np.log(s) - 0.5 * np.log(2 * np.pi) - 0.5 * ((obs - f) / s) ** 2).sum(-1)


@pytest.mark.parametrize("nlc,per,ns,npb,k0", CASES)
def test_lnl_and_gradient(nlc, per, ns, npb, k0):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    data, prm, obs, sigma = problem(nlc, per, ns, npb, k0)
    m = RoadRunnerModel('quadratic')
    m.set_data(**data)
    ref = oracle.OracleRoadRunner('quadratic')
    ref.set_data(**data)
    args = lambda q: tuple(q[n] for n in ('k', 'ldc', 't0', 'p', 'a', 'i', 'e', 'w'))
    lnl, g = lnlikelihood(m, obs, sigma, *args(prm), grad=True)
    np.testing.assert_allclose(lnl, oracle_lnl(ref, data, prm, obs, sigma), rtol=1e-9)
    np.testing.assert_array_equal(lnl, lnlikelihood(m, obs, sigma, *args(prm)))
    g2 = lnlikelihood(m, obs, sigma, *args(prm), grad=True)[1]
    np.testing.assert_array_equal(g, g2)   # bit for bit
    ms = RoadRunnerModel('quadratic', precision='split')
    ms.set_data(**data)
    gs = lnlikelihood(ms, obs, sigma, *args(prm), grad=True)[1]
    assert (np.abs(g - gs).max(0) <= 1e-4 * np.abs(g).max(0)).all()
