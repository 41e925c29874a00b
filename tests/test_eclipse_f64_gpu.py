"""The FP64 eclipse and eclipse-spectroscopy kernels at the sizes where they
change form, against the oracle.

Tolerance 2e-13 absolute: the eclipse time's rounding (~2e-15 d, another
library's sines) times the sky speed (up to 25 stellar radii a day) and the
closed form of the orbit against Newton's method on Kepler's equation (2e-15
of terms up to five) move z by at most 6e-14, and the area by at most 2
sin(kappa1) <= 2 times that; the area's own rounding is below 1e-15.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 2e-13


def close(got, want):
    assert got.shape == want.shape and np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.abs(got[ok] - want[ok]).max() <= TOL


@pytest.mark.parametrize("k", [1e-7, 0.01, 0.1, 0.25, 0.6, 0.999, 1.0, 1.4])
@pytest.mark.parametrize("b,ecc,ns", [(0.0, 0.0, 1), (0.3, 0.2, 3), (0.97, 0.0, 300)])
def test_eclipse_areas(k, b, ecc, ns):
    from pytransit_gb300 import EclipseModel
    npv = 3
    p, a = np.array([3.0, 2.0, 5.0]), np.array([8.0, 5.0, 11.0])
    a_bad = a.copy()
    a_bad[1] = 0.5
    w = np.array([0.3, 2.0, 5.0])
    t0 = np.zeros((npv, 1))
    time = np.concatenate([c + np.linspace(-0.2, 0.2, 301) for c in (0.0, 1.5, 3.0)])
    m = EclipseModel()
    m.set_data(time, nsamples=[ns], exptimes=[0.02 if ns > 1 else 0.0])
    args = (np.full(npv, k), t0, p, a_bad, np.arccos(b / a), np.full(npv, ecc), w)
    m.fp64_cull = False
    plain = m.evaluate(*args, copy=False).cpu().numpy()
    m.fp64_cull = True
    got = m.evaluate(*args, copy=False).cpu().numpy()
    np.testing.assert_array_equal(got, plain)
    want = oracle.eclipse_full(time, *args, 1.0, np.zeros(time.size, int), [0], [ns], [0.02 if ns > 1 else 0.0])
    assert np.isnan(want[1]).all()
    close(got, want)


@pytest.mark.parametrize("npv,npt,npb,ns,ecc", [(1, 1, 1, 1, 0.0), (1, 33, 3, 2, 0.0), (3, 500, 513, 1, 0.2),
                                                (5, 4001, 2, 300, 0.1), (700, 3000, 4, 1, 0.0)])
def test_es(npv, npt, npb, ns, ecc):
    from pytransit_gb300 import ESModel
    rng = np.random.default_rng(npt)
    p, a = rng.uniform(1.0, 4.0, npv), rng.uniform(4.0, 12.0, npv)
    if npv > 2:
        a[2] = 0.9
    time = np.arange(npt) * (0.004 if npt > 40 else 0.05)
    prm = (rng.uniform(0.05, 0.2, npv), rng.normal(0.0, 1e-2, npv), p, a,
           np.arccos(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0)), rng.uniform(0, ecc, npv), rng.uniform(0, 6, npv))
    f = rng.uniform(1e-4, 5e-3, (npv, npb))
    m = ESModel()
    m.set_data(time, nsamples=[ns], exptimes=[0.01 if ns > 1 else 0.0])
    got = m.evaluate(f, *prm, rstar=0.8, copy=False).cpu().numpy()
    want = oracle.es_full(time, *prm, np.full(npv, 0.8), f, ns, 0.01 if ns > 1 else 0.0)
    close(got, want.reshape(got.shape))
