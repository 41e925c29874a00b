"""The split likelihood and its adjoint around the number of samples kept
between its two passes (8), with a thread's points in one and in several light
curves, some of them out of transit altogether.

lnL against the FP64 kernels, to what 1e-6 in the flux allows; the same bits
with and without the gradient and on a second run.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("nlc,per,npb,k0", [(1, 3000, 1, 0.1), (7, 150, 2, 0.15), (70, 20, 1, 0.6), (2, 500, 2, 1.2)])
def test_against_fp64(ns, nlc, per, npb, k0):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(ns + nlc)
    npv = 4
    time = np.concatenate([1.5 * j + np.linspace(-0.15, 0.12, per) for j in range(nlc)])   # every other one in transit
    data = dict(time=time, lcids=np.repeat(np.arange(nlc), per), pbids=np.arange(nlc) % npb, nsamples=[ns] * nlc,
                exptimes=[0.02 if ns > 1 else 0.0] * nlc)
    a = rng.uniform(6, 12, npv)
    prm = (k0 * rng.uniform(0.9, 1.1, (npv, npb)), rng.uniform(0.1, 0.4, (npv, npb, 2)), rng.normal(0, 1e-3, (npv, 1)),
           3.0 + rng.normal(0, 1e-3, npv), a, np.arccos(rng.uniform(0.1, 0.8, npv) / a), rng.uniform(0.05, 0.2, npv),
           rng.uniform(0, 6, npv))
    obs, sigma = 1.0 + rng.normal(0, 1e-3, time.size), 1e-3
    out = {}
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel('quadratic', precision=precision)
        m.set_data(**data)
        lnl, g = lnlikelihood(m, obs, sigma, *prm, grad=True)
        out[precision] = lnl
        np.testing.assert_array_equal(lnl, lnlikelihood(m, obs, sigma, *prm))
        np.testing.assert_array_equal(g, lnlikelihood(m, obs, sigma, *prm, grad=True)[1])
        if precision == 'fp64':
            r = np.abs(obs - m.evaluate(*prm).reshape(npv, -1)).sum(1)
    assert (np.abs(out['split'] - out['fp64']) <= 1e-6 * (r + time.size * 1e-6) / sigma ** 2).all()
