"""Limb-darkening means and their derivatives from weight tables whose rows are
and are not whole 16-byte words, small and too large to be staged, at radius
ratios inside and outside the table, with fewer and more passbands than a block
takes at once.

Flux of the split path against the FP64 path to 1e-6, and of the FP64 path
against the oracle to 1e-9; the likelihood's derivatives with respect to the
radius ratios and limb darkening to 1e-4 of each column's largest value (sums
of terms of one sign: the data have no transit, so every residual is a deficit).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nzin,nzlimb", [(20, 20), (20, 22), (21, 20), (2, 1), (30, 34)])
@pytest.mark.parametrize("ng", [50, 100, 230])
@pytest.mark.parametrize("npb,k0", [(1, 0.1), (6, 0.12), (1, 0.6)])
def test_means(nzin, nzlimb, ng, npb, k0):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(nzin + ng + npb)
    npv, per = 5, 120
    kw = dict(nzin=nzin, nzlimb=nzlimb, ng=ng, nk=64, klims=(0.05, 0.2))
    data = dict(time=np.tile(np.linspace(-0.1, 0.09, per), npb), lcids=np.repeat(np.arange(npb), per), pbids=np.arange(npb))
    a = rng.uniform(6, 12, npv)
    prm = (k0 * rng.uniform(0.9, 1.1, (npv, npb)), rng.uniform(0.3, 0.8, (npv, npb, 2)), rng.normal(0, 1e-3, npv),
           np.full(npv, 3.0), a, np.arccos(rng.uniform(0.1, 0.6, npv) / a), rng.uniform(0, 0.1, npv), rng.uniform(0, 6, npv))
    ref = oracle.OracleRoadRunner('power-2', **kw)
    ref.set_data(**data)
    out = {}
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel('power-2', precision=precision, **kw)
        m.set_data(**data)
        g = lnlikelihood(m, np.ones(data['time'].size), 1e-3, *prm, grad=True)[1]
        out[precision] = m.evaluate(*prm).reshape(npv, -1), g[:, np.r_[0:npb, npb + 6:g.shape[1]]]
    (f64, g64), (f32, g32) = out['fp64'], out['split']
    np.testing.assert_allclose(f64, ref.evaluate(*prm).reshape(npv, -1), rtol=1e-9)
    assert np.abs(f32 - f64).max() <= 1e-6
    assert (np.abs(g32 - g64).max(0) <= 1e-4 * np.abs(g64).max(0)).all()
