"""Error bounds of the split transmission-spectroscopy path do not depend on how
many parameter vectors share the launch: few (a block of warps for each), many
(four to a block, the last block partial), one channel up to more than a
block's warps, an invalid vector among them.  The same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npb", [1, 7, 33, 70])
def test_bounds_of_any_population(npb):
    from pytransit_gb300 import TSModel
    rng = np.random.default_rng(npb)
    npv = 1025
    a = rng.uniform(3, 15, npv)
    a[[0, 600]] = 0.8
    args = (rng.uniform(0.05, 0.2, (npv, npb)), rng.uniform(0.1, 0.4, (npv, npb, 2)), rng.normal(0, 1e-3, npv),
            rng.uniform(1, 5, npv), a, np.arccos(rng.uniform(0, 0.8, npv) / np.maximum(a, 1)), rng.uniform(0, 0.2, npv),
            rng.uniform(0, 6, npv))
    m = TSModel('quadratic', precision='split')
    m.set_data(np.linspace(-0.1, 0.1, 20), nsamples=[3], exptimes=[0.01])
    m.evaluate(*args, return_error=True)
    whole = m.error_bounds()
    parts = []
    for lo, hi in ((0, 1), (1, 4), (4, 9), (9, 500), (500, 1025)):
        m.evaluate(*(x[lo:hi] for x in args), return_error=True)
        parts.append(m.error_bounds())
    assert np.array_equal(whole, np.concatenate(parts))
    assert (whole > 0).sum() == npv - 2
