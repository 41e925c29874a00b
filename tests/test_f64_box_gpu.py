"""The edges of the FP64 models' bounding box where they cut through a transit:
a box that belongs to the first of several radius ratios, a grazing first one, an
orbit so close that the contact is outside the bisection's bracket.  Points from
3e-9 d on either side of the oracle's edges, where the flux jumps by up to k^2.
Against the oracle: 1e-9 (2e-13 for eclipses), the paths' tolerances, and
no point on the other side of an edge.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

OFF = np.array([3e-9, 3e-8, 1e-7, 2e-7, 5e-7, 1e-6, 1e-5])
OFF = np.concatenate([-OFF[::-1], OFF])


def edges(k0, p, a, inc, e, w, pad):
    t1, t4 = oracle.bounding_box(k0, np.asarray(oracle.solve2d(0.0, p, a, inc, e, w)).ravel())
    return np.concatenate([t1 - pad + OFF, t4 + pad + OFF, np.linspace(t1, t4, 7)])


# first and second radius ratio, period, a, impact parameter, e
ORBITS = [(0.05, 0.2, 9.0, 6.0, 0.3, 0.0), (0.05, 0.2, 9.0, 6.0, 0.9, 0.2), (0.02, 0.4, 30.0, 9.0, 0.5, 0.1),
          (0.05, 0.3, 12.0, 5.0, 1.05, 0.0),           # grazing by its end, t1 = 0 nearly
          (0.0499999, 0.3, 12.0, 5.0, 1.05, 0.0), (0.05, 0.3, 12.0, 5.0, 1.06, 0.0),   # out of transit: whole bracket
          (1.2, 1.3, 5.0, 1.3, 0.2, 0.0), (0.9, 0.9, 8.0, 1.05, 0.1, 0.0)]


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("orbit", ORBITS)
def test_transit(orbit, ns):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    k0, k1, p, a, b, e = orbit
    inc, w, ex = np.arccos(b / a), 1.0, 0.02 if ns > 1 else 0.0
    t = edges(k0, p, a, inc, e, w, 0.003 + ex)
    data = dict(time=np.tile(t, 2), lcids=np.repeat([0, 1], t.size), pbids=[0, 1], nsamples=[ns] * 2, exptimes=[ex] * 2)
    args = ([[k0, k1]], [[[0.4, 0.2]] * 2], 0.0, p, a, inc, e, w)
    ref = oracle.OracleRoadRunner('quadratic')
    ref.set_data(**data)
    want = ref.evaluate(*args)
    m = RoadRunnerModel('quadratic')
    m.set_data(**data)
    for cull in (False, True):
        m.fp64_cull = cull
        got = m.evaluate(*args, copy=False).cpu().numpy()
        assert np.abs(got - want).max() <= 1e-9
    obs = np.ones(2 * t.size)
    lnl = lnlikelihood(m, obs, 1e-3, *args)
    np.testing.assert_allclose(lnl, oracle.lnlike_normal(obs, want[None, :], 1e-3), rtol=1e-9)
    np.testing.assert_allclose(lnlikelihood(m, obs, 1e-3, *args, grad=True)[0], lnl, rtol=0, atol=0)


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("orbit", [(1.2, 5.0, 1.3, 0.2), (0.9, 8.0, 1.05, 0.1), (0.1, 3.0, 8.0, 0.3)])
def test_transmission_spectroscopy(orbit, ns):
    from pytransit_gb300 import TSModel
    k0, p, a, b = orbit
    inc, ex, npb = np.arccos(b / a), 0.02 if ns > 1 else 0.0, 6
    t = edges(k0, p, a, inc, 0.0, 0.0, 0.0015 + ex)
    ref = oracle.OracleRoadRunner('quadratic', ts=True)
    ref.set_data(t, nsamples=[ns], exptimes=[ex])
    m = TSModel('quadratic')
    m.set_data(t, nsamples=[ns], exptimes=[ex])
    args = (np.full((1, npb), k0), np.tile([0.4, 0.2], (1, npb, 1)), np.zeros(1), p, a, inc, 0.0, 0.0)
    got = m.evaluate(*args)
    assert np.abs(got - ref.evaluate(*args).reshape(got.shape)).max() <= 1e-9


@pytest.mark.parametrize("ns", [1, 3])
@pytest.mark.parametrize("orbit", [(1.2, 5.0, 1.3, 0.2), (0.9, 8.0, 1.05, 0.1), (0.1, 3.0, 8.0, 0.3)])
def test_eclipse(orbit, ns):
    from pytransit_gb300 import EclipseModel, EclipseSpectroscopyModel
    k, p, a, b = orbit
    inc, ex, light = np.arccos(b / a), 0.02 if ns > 1 else 0.0, 6.957e8 / 299792458.0 / 86400.0
    te = 0.5 * p + 2 * a * np.sin(inc) * light
    prm = tuple(np.array([v]) for v in (p, a, inc, 0.0, 0.0))
    for pad in (0.003, 0.0015):
        # the edges' own times are rounded at te: stay 1e-12 d away from them
        t = te + edges(k, p, a, inc, 0.0, 0.0, pad + ex)
        if pad == 0.003:
            want = oracle.eclipse_full(t, np.array([k]), np.zeros((1, 1)), *prm, 1.0, np.zeros(t.size, int), [0], [ns], [ex])
            m = EclipseModel()
            m.set_data(t, nsamples=[ns], exptimes=[ex])
            got = m.evaluate(np.array([k]), np.zeros((1, 1)), *prm, copy=False).cpu().numpy()
        else:
            f = np.array([[0.3, 0.5]])
            want = oracle.es_full(t, np.array([k]), np.zeros(1), *prm, np.ones(1), f, ns, ex)
            m = EclipseSpectroscopyModel()
            m.set_data(t, nsamples=[ns], exptimes=[ex])
            got = m.evaluate(f, np.array([k]), np.zeros(1), *prm, copy=False).cpu().numpy()
        assert np.abs(got - np.asarray(want).reshape(got.shape)).max() <= 2e-13
