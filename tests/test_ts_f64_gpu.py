"""The FP64 transmission-spectroscopy path for the affine laws (basis columns
instead of a LD-mean table per channel) against the general path, which the
same profile takes when it is given as a user callable, and its launch shapes.

Tolerance 1e-13: both take the same overlap areas; the order of the sums over
the weight table's columns, the samples and the basis functions differs, a
few tens of roundings of terms below one.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def profiles():
    from pytransit_gb300 import ldmodels as ld
    return {n: (e if isinstance(e, tuple) else (e, None)) for n, e in ld.NAMED_LAWS.items()}


COEF = {'uniform': 0, 'linear': 1, 'quadratic': 2, 'quadratic-tri': 2, 'nonlinear': 4, 'square_root': 2}


@pytest.mark.parametrize("law", list(COEF))
@pytest.mark.parametrize("npv,npb,npt,ns,k0", [(1, 1, 1, 1, 0.1), (2, 3, 130, 1, 0.1), (3, 6, 257, 3, 0.1),
                                               (4, 65, 500, 40, 0.2), (3, 200, 301, 2, 0.6), (2, 7, 200, 2, 1.1)])
def test_basis_columns_match_the_general_path(law, npv, npb, npt, ns, k0):
    from pytransit_gb300 import TSModel
    if law not in profiles():
        pytest.skip("law not in this build")
    rng = np.random.default_rng(npb)
    fl, fi = profiles()[law]
    wrap = (lambda mu, pv: fl(mu, pv)) if fi is None else (lambda mu, pv: fl(mu, pv), lambda pv: fi(pv))
    ldc = rng.uniform(0.05, 0.3, (npv, npb, max(1, COEF[law])))
    a = rng.uniform(4, 12, npv)
    if npv > 2:
        a[1] = 0.7
    args = (k0 * rng.uniform(0.9, 1.1, (npv, npb)), ldc, rng.normal(0, 1e-3, npv), rng.uniform(2, 5, npv), a,
            np.arccos(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0)), rng.uniform(0, 0.2, npv), rng.uniform(0, 6, npv))
    out = []
    for model in (law, wrap):
        m = TSModel(model)
        m.set_data(np.linspace(-0.15, 0.15, npt) if npt > 1 else np.array([0.01]), nsamples=[ns],
                   exptimes=[0.01 if ns > 1 else 0.0])
        out.append(m.evaluate(*args, copy=False).cpu().numpy())
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    ok = ~np.isnan(out[0])
    assert (out[0][ok] < 1.0).any() or npt == 1
    assert np.abs(out[0][ok] - out[1][ok]).max() <= 1e-13
