"""FP64 profiles and disk integrals of the affine laws without a closed-form
integral, from sums shared by a block's passbands: one passband up to several
blocks of them (16 each, the last partial), grids up to the largest staged.

Flux against the oracle (the profile at every point, the 200-point trapezoid per
passband) to 1e-9; a NaN coefficient gives NaN for its own vector alone.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NPAR = {'nonlinear': 4, 'square_root': 2, 'general': 3}


@pytest.mark.parametrize("law", list(NPAR))
@pytest.mark.parametrize("npv,npb,nz", [(1, 1, 40), (5, 3, 40), (16, 1, 3), (33, 2, 64), (70, 1, 41)])
def test_against_the_oracle(law, npv, npb, nz):
    from pytransit_gb300 import RoadRunnerModel
    rng = np.random.default_rng(npv)
    kw = dict(nzin=nz // 2, nzlimb=nz - nz // 2, nk=64)
    try:
        m = RoadRunnerModel(law, **kw)
    except ValueError:
        pytest.skip("law not in this build")
    ref = oracle.OracleRoadRunner(law, **kw)
    per = 60
    data = dict(time=np.tile(np.linspace(-0.1, 0.1, per), npb), lcids=np.repeat(np.arange(npb), per), pbids=np.arange(npb))
    a = rng.uniform(5, 12, npv)
    ldc = rng.uniform(0.05, 0.3, (npv, npb, NPAR[law]))
    args = (rng.uniform(0.06, 0.14, (npv, npb)), ldc, rng.normal(0, 1e-3, npv), np.full(npv, 3.0), a,
            np.arccos(rng.uniform(0, 0.7, npv) / a), rng.uniform(0, 0.2, npv), rng.uniform(0, 6, npv))
    m.set_data(**data)
    ref.set_data(**data)
    got = m.evaluate(*args).reshape(npv, -1)
    np.testing.assert_allclose(got, ref.evaluate(*args).reshape(npv, -1), rtol=0, atol=1e-9)
    bad = ldc.copy()
    bad[-1, 0, -1] = np.nan
    out = m.evaluate(args[0], bad, *args[2:]).reshape(npv, -1)
    assert np.array_equal(out[:-1], got[:-1]) and np.isnan(out[-1]).any()
