"""NaN parameters in the FP64 flux, log-likelihood and adjoint: such a vector
takes the reference's NaN (in the box) and 1 (out of it), its log-likelihood
and gradient are NaN, and the other vectors keep their bits.  Against the
oracle, whose table lookup is checked on the host first.
"""
import numpy as np
import pytest

import oracle

LAW = 'quadratic'
TOL = 1e-9      # the FP64 path's


def test_oracle_interpolation_of_nan():
    """A NaN position has no table index."""
    lda = np.ones(100)
    assert np.isnan(oracle.interp_ldm(float('nan'), 0.01, lda))
    assert np.isnan(oracle.interp_ldm(-1e-3, 0.01, lda))
    assert oracle.interp_ldm(1.5, 0.01, lda) == 0.0


def problem(npt, ns, npb):
    rng = np.random.default_rng(npt + ns)
    npv, nlc = 5, npb
    time = np.concatenate([3.0 * j + np.linspace(-0.3, 0.3, npt) for j in range(nlc)])
    data = dict(time=time, lcids=np.repeat(np.arange(nlc), npt), pbids=np.arange(nlc), nsamples=[ns] * nlc,
                exptimes=[0.02 if ns > 1 else 0.0] * nlc)
    a = rng.uniform(8, 12, npv)
    prm = dict(k=rng.uniform(0.08, 0.12, (npv, npb)), ldc=rng.uniform(0.1, 0.4, (npv, npb, 2)),
               t0=rng.normal(0, 1e-3, (npv, 1)), p=np.full(npv, 3.0), a=a, i=np.arccos(rng.uniform(0.1, 0.8, npv) / a),
               e=rng.uniform(0.05, 0.2, npv), w=rng.uniform(0, 6, npv))
    return data, prm


def args(prm):
    return tuple(prm[n] for n in ('k', 'ldc', 't0', 'p', 'a', 'i', 'e', 'w'))


# NaN k, i: NaN in the box; the others move the box away, and every point is 1
NAN = ['k', 'i', 'p', 't0', 'e', 'w']


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAN)
@pytest.mark.parametrize("npt,ns,npb", [(300, 1, 1), (300, 3, 1), (300, 2, 2)])
def test_flux(name, npt, ns, npb):
    from pytransit_gb300 import RoadRunnerModel
    data, good = problem(npt, ns, npb)
    prm = {n: v.copy() for n, v in good.items()}
    prm[name][2] = np.nan
    if name == 'k' and npb > 1:
        prm['k'][4, 1] = np.nan          # the second passband alone: the box is that of the first
    ref = oracle.OracleRoadRunner(LAW)
    ref.set_data(**data)
    want = ref.evaluate(*args(prm))
    assert np.isnan(want[2]).any() == (name in 'ki')
    m = RoadRunnerModel(LAW)
    m.set_data(**data)
    for cull in (False, True):
        m.fp64_cull = cull
        got = m.evaluate(*args(prm), copy=False).cpu().numpy()
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        ok = ~np.isnan(want)
        assert np.abs(got[ok] - want[ok]).max() <= TOL
        np.testing.assert_array_equal(got[[0, 1, 3]], m.evaluate(*args(good), copy=False).cpu().numpy()[[0, 1, 3]])


@pytest.mark.gpu
@pytest.mark.parametrize("name", NAN)
@pytest.mark.parametrize("npt,ns,npb", [(300, 1, 1), (300, 3, 1), (300, 2, 2)])
def test_lnlikelihood(name, npt, ns, npb):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    data, good = problem(npt, ns, npb)
    prm = {n: v.copy() for n, v in good.items()}
    prm[name][2] = np.nan
    obs = 1.0 + np.random.default_rng(1).normal(0, 1e-3, data['time'].size)
    m = RoadRunnerModel(LAW)
    m.set_data(**data)
    lnl0, g0 = lnlikelihood(m, obs, 1e-3, *args(good), grad=True)
    lnl, g = lnlikelihood(m, obs, 1e-3, *args(prm), grad=True)
    flux = m.evaluate(*args(prm))
    assert np.isnan(lnl[2]) == np.isnan(flux[2]).any() == (name in 'ki')
    assert np.isnan(g[2]).all() == (name in 'ki')
    rest = [0, 1, 3, 4]
    np.testing.assert_array_equal(lnl[rest], lnl0[rest])
    np.testing.assert_array_equal(g[rest], g0[rest])
    np.testing.assert_array_equal(lnlikelihood(m, obs, 1e-3, *args(prm)), lnl)


@pytest.mark.gpu
def test_walker_with_negative_area_ratio():
    """k = sqrt(k2) of a sampler's walker outside the prior."""
    import torch
    from pytransit_gb300 import RoadRunnerModel, lpf
    rng = np.random.default_rng(3)
    time = np.linspace(-0.1, 0.1, 500)
    m = RoadRunnerModel(LAW)
    m.set_data(time)
    pv = np.tile([0.0, 3.0, 1.4, 0.3, 0.01, 0.4, 0.3], (4, 1))
    obs = torch.as_tensor(1.0 + rng.normal(0, 1e-3, time.size)).cuda()
    good = lpf.lnlikelihood(m, obs, 1e-3, torch.as_tensor(pv).cuda(), 0.0).cpu().numpy()
    pv[1, 4] = -0.01
    got = lpf.lnlikelihood(m, obs, 1e-3, torch.as_tensor(pv).cuda(), 0.0).cpu().numpy()
    assert np.isnan(got[1])
    np.testing.assert_array_equal(got[[0, 2, 3]], good[[0, 2, 3]])


@pytest.mark.gpu
@pytest.mark.parametrize("name", ['k', 'i', 'w', 'p'])
@pytest.mark.parametrize("ns", [1, 3])
def test_eclipses(name, ns):
    from pytransit_gb300 import EclipseModel, EclipseSpectroscopyModel
    npv, time = 3, np.concatenate([np.linspace(-0.2, 0.2, 200), 1.5 + np.linspace(-0.4, 0.4, 400)])
    a = np.array([8.0, 5.0, 11.0])
    prm = dict(k=np.full(npv, 0.1), t0=np.zeros(npv), p=np.full(npv, 3.0), a=a, i=np.arccos(0.3 / a),
               e=np.full(npv, 0.1), w=np.array([0.3, 2.0, 5.0]))
    prm[name][1] = np.nan
    order = tuple(prm[n] for n in ('k', 't0', 'p', 'a', 'i', 'e', 'w'))
    ex = 0.02 if ns > 1 else 0.0
    want = oracle.eclipse_full(time, order[0], prm['t0'].reshape(npv, 1), *order[2:], 1.0, np.zeros(time.size, int), [0],
                               [ns], [ex])
    m = EclipseModel()
    m.set_data(time, nsamples=[ns], exptimes=[ex])
    for cull in (False, True):
        m.fp64_cull = cull
        np.testing.assert_allclose(m.evaluate(order[0], prm['t0'].reshape(npv, 1), *order[2:], copy=False).cpu().numpy(),
                                   want, rtol=0, atol=2e-13)
    f = np.full((npv, 2), 1e-3)
    want = oracle.es_full(time, *order, np.ones(npv), f, ns, ex)
    m = EclipseSpectroscopyModel()
    m.set_data(time, nsamples=[ns], exptimes=[ex])
    got = m.evaluate(f, *order, copy=False).cpu().numpy()
    np.testing.assert_allclose(got, want.reshape(got.shape), rtol=0, atol=2e-13)


@pytest.mark.gpu
@pytest.mark.parametrize("w", [np.nan, np.inf])
def test_argument_of_periastron_of_a_circular_orbit(w):
    """e = 0 does not hide a w that is no angle: e sin w is NaN."""
    from pytransit_gb300 import EclipseModel, RoadRunnerModel, TSModel
    from pytransit_gb300.lnlike import lnlikelihood
    data, prm = problem(300, 1, 1)
    prm['e'][:] = 0.0
    prm['w'][2] = w
    ref = oracle.OracleRoadRunner(LAW)
    ref.set_data(**data)
    want = ref.evaluate(*args(prm))
    assert (want[2] == 1.0).all() and (want[1] < 1.0).any()
    m = RoadRunnerModel(LAW)
    m.set_data(**data)
    np.testing.assert_allclose(m.evaluate(*args(prm)), want, rtol=0, atol=TOL)
    obs = np.ones(300)
    np.testing.assert_allclose(lnlikelihood(m, obs, 1e-3, *args(prm)), oracle.lnlike_normal(obs, want, 1e-3), rtol=1e-9)
    ref = oracle.OracleRoadRunner(LAW, ts=True)
    ref.set_data(data['time'])
    m = TSModel(LAW)
    m.set_data(data['time'])
    prm['t0'] = prm['t0'][:, 0]
    got = m.evaluate(*args(prm))
    np.testing.assert_allclose(got, ref.evaluate(*args(prm)).reshape(got.shape), rtol=0, atol=TOL)
    order = (prm['k'][:, 0], prm['t0'].reshape(-1, 1), *(prm[n] for n in ('p', 'a', 'i', 'e', 'w')))
    time = np.linspace(1.2, 1.8, 200)
    m = EclipseModel()
    m.set_data(time)
    np.testing.assert_allclose(m.evaluate(*order), oracle.eclipse_full(time, *order, 1.0, np.zeros(200, int), [0], [1], [0.0]),
                               rtol=0, atol=2e-13)
