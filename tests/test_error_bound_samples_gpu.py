"""The stated error bound with large exposures and fast orbits, where the sample
times' roundings are a large part of it: at least the measured error against the
FP64 path for every parameter vector, by each way a supersampled light curve takes
(long ones, short ones, points of several interleaved), and for transmission
spectroscopy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def population(rng, npv):
    a = rng.uniform(1.5, 4.0, npv)
    return dict(p=rng.uniform(0.3, 0.8, npv), a=a, i=np.arccos(rng.uniform(0, 0.9, npv) / a), e=rng.uniform(0, 0.1, npv),
                w=rng.uniform(0, 2 * np.pi, npv))


@pytest.mark.parametrize("ns", [2, 7, 12, 300])
@pytest.mark.parametrize("exposure", [0.02, 0.15])
@pytest.mark.parametrize("layout", ["long", "short", "interleaved"])
def test_light_curves(ns, exposure, layout):
    from pytransit_gb300 import RoadRunnerModel
    rng = np.random.default_rng(ns)
    npv, npt = 200, 1500
    nlc = {"long": 1, "short": 12, "interleaved": 2}[layout]
    lcids = np.arange(npt) % 2 if layout == "interleaved" else np.arange(npt) * nlc // npt
    prm = population(rng, npv)
    args = (rng.uniform(0.05, 0.4, (npv, 1)), rng.uniform(0.1, 0.4, (npv, 1, 2)), rng.normal(0, 1e-2, (npv, 1)),
            *(prm[n] for n in ('p', 'a', 'i', 'e', 'w')))
    out = {}
    for precision in ('split', 'fp64'):
        m = RoadRunnerModel('quadratic', precision=precision)
        m.set_data(np.arange(npt) * 0.0021, lcids=lcids, pbids=np.zeros(nlc, int), nsamples=[ns] * nlc,
                   exptimes=[exposure] * nlc)
        out[precision] = m.evaluate(*args, copy=False).double().cpu().numpy(), m.error_bounds()
    err = np.abs(out['split'][0] - out['fp64'][0]).max(1)
    assert (err <= out['split'][1]).all() and (out['split'][1] < 1e-4).all()


@pytest.mark.parametrize("ns", [1, 2, 7, 300])
def test_transmission_spectroscopy(ns):
    from pytransit_gb300 import TSModel
    rng = np.random.default_rng(ns)
    npv, npb = 60, 8
    prm = population(rng, npv)
    args = (rng.uniform(0.09, 0.11, (npv, npb)), rng.uniform(0.1, 0.4, (npv, npb, 2)), rng.normal(0, 1e-2, npv),
            *(prm[n] for n in ('p', 'a', 'i', 'e', 'w')))
    out = {}
    for precision in ('split', 'fp64'):
        m = TSModel('quadratic', precision=precision)
        m.set_data(np.arange(700) * 0.0041, nsamples=[ns], exptimes=[0.1 if ns > 1 else 0.0])
        out[precision] = m.evaluate(*args, copy=False).double().cpu().numpy(), m.error_bounds()
    err = np.abs(out['split'][0] - out['fp64'][0]).max((1, 2))
    assert (err <= out['split'][1]).all()
