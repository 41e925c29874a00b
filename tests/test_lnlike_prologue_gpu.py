"""The FP64 likelihood on the fused prologue of the affine laws against the
general one (LD means from the weight tables), radius ratios inside and outside
the table, one and several passbands, with and without the gradient.

Relative 1e-11 on lnL and 1e-10 of each gradient column's largest value: the LD
means differ by the order of sums of a few tens of terms below one (1e-15),
lnL and the gradient weight them with (o - m) / sigma^2 of 1e3 to 1e6 over their
own sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law,nc", [('uniform', 0), ('linear', 1), ('quadratic', 2), ('quadratic-tri', 2), ('nonlinear', 4),
                                    ('power-2', 2)])
@pytest.mark.parametrize("npv,npb", [(1, 1), (33, 3)])
def test_fused_against_general(law, nc, npv, npb, monkeypatch):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(nc + npv)
    per = 150
    m = RoadRunnerModel(law, nk=64, klims=(0.05, 0.2))
    m.set_data(np.tile(np.linspace(-0.12, 0.1, per), npb), lcids=np.repeat(np.arange(npb), per), pbids=np.arange(npb))
    a = rng.uniform(5, 12, npv)
    k = rng.uniform(0.06, 0.18, (npv, npb))
    k[-1] = 0.3
    args = (k, rng.uniform(0.1, 0.3, (npv, npb, nc)), rng.normal(0, 1e-3, npv), np.full(npv, 3.0), a,
            np.arccos(rng.uniform(0, 0.7, npv) / a), rng.uniform(0, 0.2, npv), rng.uniform(0, 6, npv))
    obs = 1 + rng.normal(0, 1e-3, per * npb)
    lnl, g = lnlikelihood(m, obs, 1e-3, *args, grad=True)
    assert np.array_equal(lnl, lnlikelihood(m, obs, 1e-3, *args))
    monkeypatch.setattr(m, '_basis', lambda *_: (None, 0))
    lnl2, g2 = lnlikelihood(m, obs, 1e-3, *args, grad=True)
    np.testing.assert_allclose(lnl, lnl2, rtol=1e-11)
    assert (np.abs(g - g2).max(0) <= 1e-10 * np.abs(g2).max(0)).all()
