"""The FP64 log-likelihood and gradient with the points of several light curves
interleaved, of one and of several passbands and epochs, at the sizes where a
tile's points of a light curve start, fill and overflow the queue.  Against
torch's automatic differentiation of the same model (1e-9 of each column, as
derived there), and the same lnL bits with and without the gradient.
"""
import numpy as np
import pytest
import torch

import oracle
from test_lnlike_gradient_gpu import model_lnl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlc,npb,nep", [(2, 1, 1), (4, 4, 2), (4, 2, 1), (40, 3, 2)])
@pytest.mark.parametrize("npt,ns", [(61, 1), (600, 1), (300, 3)])
def test_interleaved(nlc, npb, nep, npt, ns):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(nlc * npt)
    npv = 3
    time = np.linspace(-0.1, 0.1, npt)
    data = dict(time=time, lcids=np.arange(npt) % nlc, pbids=np.arange(nlc) % npb, nsamples=[ns] * nlc,
                exptimes=[0.01 if ns > 1 else 0.0] * nlc, epids=(np.arange(nlc) // 2) % nep)
    a = rng.uniform(6, 12, npv)
    prm = dict(k=rng.uniform(0.08, 0.12, (npv, npb)), t0=rng.normal(0, 1e-3, (npv, nep)), p=3.0 + rng.normal(0, 1e-4, npv),
               a=a, i=np.arccos(rng.uniform(0.1, 0.8, npv) / a), e=rng.uniform(0.05, 0.2, npv), w=rng.uniform(0, 6, npv),
               ldc=rng.uniform(0.1, 0.4, (npv, npb, 2)))
    sigma = rng.uniform(0.8e-3, 1.2e-3, nlc)
    obs = 1.0 - 0.008 * (np.abs(time) < 0.06) + rng.normal(0, 1e-3, npt)
    ref = oracle.OracleRoadRunner('quadratic')
    x = {n: torch.as_tensor(v).requires_grad_(True) for n, v in prm.items()}
    want = model_lnl(ref, data, obs, sigma, *(x[n] for n in ('k', 't0', 'p', 'a', 'i', 'e', 'w', 'ldc')))
    gw = torch.autograd.grad(want.sum(), list(x.values()))
    gw = np.concatenate([v.reshape(npv, -1).numpy() for v in gw], 1)
    m = RoadRunnerModel('quadratic')
    m.set_data(**data)
    args = tuple(prm[n] for n in ('k', 'ldc', 't0', 'p', 'a', 'i', 'e', 'w'))
    lnl, g = lnlikelihood(m, obs, sigma, *args, grad=True)
    np.testing.assert_allclose(lnl, want.detach().numpy(), rtol=1e-10)
    scale = np.abs(gw).max(0)
    # the period's column vanishes: every point is of epoch 0, and its share through the orbit is small
    assert (np.abs(g - gw).max(0) <= 1e-9 * scale + 1e-13 * scale.max()).all()
    np.testing.assert_array_equal(lnlikelihood(m, obs, sigma, *args), lnl)
