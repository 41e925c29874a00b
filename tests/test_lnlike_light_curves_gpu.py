"""The FP64 likelihood's change from one light curve to the next inside a warp's
share of a row: light curves of a few points, so that each flush of the queue
is another light curve's, also beyond the light curves a block stages.  Sums
bit for bit the same in every run, and the light curves' own likelihoods add
up to the whole (1e-12 of the terms' sum: each is a sum of a few hundred
FP64 terms).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlc,per", [(2, 40), (37, 5), (70, 3), (40, 33)])
def test_light_curves_add_up(nlc, per):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(nlc)
    npv = 40
    time = np.concatenate([3.0 * j + np.linspace(-0.05, 0.05, per) for j in range(nlc)])
    a = rng.uniform(8, 12, npv)
    args = (rng.uniform(0.08, 0.12, (npv, 1)), rng.uniform(0.1, 0.4, (npv, 1, 2)), rng.normal(0, 1e-3, (npv, 1)),
            np.full(npv, 3.0), a, np.arccos(rng.uniform(0.1, 0.8, npv) / a), np.zeros(npv), np.zeros(npv))
    obs = 1.0 + rng.normal(0, 1e-3, time.size)
    sigma = rng.uniform(0.8e-3, 1.2e-3, nlc)
    lcids = np.repeat(np.arange(nlc), per)
    m = RoadRunnerModel('quadratic')
    m.set_data(time, lcids=lcids, pbids=np.zeros(nlc, int), nsamples=[1] * nlc, exptimes=[0.0] * nlc)
    lnl, g = lnlikelihood(m, obs, sigma, *args, grad=True)
    for _ in range(5):
        lnl2, g2 = lnlikelihood(m, obs, sigma, *args, grad=True)
        np.testing.assert_array_equal(lnl2, lnl)
        np.testing.assert_array_equal(g2, g)
        np.testing.assert_array_equal(lnlikelihood(m, obs, sigma, *args), lnl)
    parts = np.zeros(npv)
    for j in range(nlc):
        one = RoadRunnerModel('quadratic')
        one.set_data(time[lcids == j])
        parts += lnlikelihood(one, obs[lcids == j], sigma[j], *args)
    np.testing.assert_allclose(parts, lnl, rtol=1e-12)
