"""The FP64 flux kernels' own sample arithmetic and work split at the sizes
where they change form: radius ratios on both sides of the kite form's range
and of the weight table, z = 0, the contacts, more samples than a queue chunk
holds, more light curves than are staged, tiles of many light curves, and the
launch's slot, tile and multi-group regimes.

Tolerance against the oracle: 1e-9 absolute flux, the FP64 path's (the weight
tables' own rounding is the largest part).  Culled and plain kernels: the same
bits.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-9


def both(data, args, law='quadratic'):
    from pytransit_gb300 import RoadRunnerModel
    m = RoadRunnerModel(law)
    m.set_data(**data)
    m.fp64_cull = False
    plain = m.evaluate(*args, copy=False).cpu().numpy()
    m.fp64_cull = True
    culled = m.evaluate(*args, copy=False).cpu().numpy()
    np.testing.assert_array_equal(culled, plain)
    ref = oracle.OracleRoadRunner(law)
    ref.set_data(**data)
    want = ref.evaluate(*args)
    assert np.array_equal(np.isnan(culled), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.abs(culled[ok] - want[ok]).max() <= TOL
    return culled


@pytest.mark.parametrize("k", [1e-7, 0.004, 0.05, 0.25, 0.4999, 0.7, 0.999, 1.0, 1.3])
@pytest.mark.parametrize("b", [0.0, 0.3, 0.95])
def test_radius_ratios_and_contacts(k, b):
    """z = 0 at the central point of a central transit; points at and within a
    few ulps of the contacts."""
    p, a = 3.0, 8.0
    inc = np.arccos(b / a)
    v = 2 * np.pi * a / p
    t = np.linspace(-0.2, 0.2, 401)
    edges = [np.sqrt(max((1 + s * k) ** 2 - b * b, 0.0)) / v for s in (-1, 1)]
    t = np.concatenate([t, *[[x, np.nextafter(x, 9), x * (1 + 1e-9), -x] for x in edges]])
    both(dict(time=t), (k, [[[0.4, 0.2]]], 0.0, p, a, inc, 0.0, 0.0))


@pytest.mark.parametrize("ns", [1, 2, 31, 256, 300])
def test_sample_counts(ns):
    rng = np.random.default_rng(ns)
    npv, t = 3, np.linspace(-0.1, 0.1, 257)
    a = rng.uniform(4, 12, npv)
    args = (rng.uniform(0.05, 0.2, (npv, 1)), np.tile([0.3, 0.2], (npv, 1, 1)), rng.normal(0, 1e-3, (npv, 1)),
            rng.uniform(2, 5, npv), a, np.arccos(rng.uniform(0, 0.9, npv) / a), rng.uniform(0, 0.3, npv),
            rng.uniform(0, 6, npv))
    both(dict(time=t, nsamples=[ns], exptimes=[0.02]), args, 'power-2')


@pytest.mark.parametrize("nlc,per", [(40, 7), (33, 129), (3, 500)])
def test_light_curves(nlc, per):
    """Tiles of up to 19 light curves, more light curves than a block stages,
    each with its own passband, epoch, exposure and sample count."""
    rng = np.random.default_rng(nlc)
    npv, npb = 4, min(nlc, 5)
    time = np.concatenate([2459000.0 + 2.0 * j + np.linspace(-0.15, 0.15, per) for j in range(nlc)])
    a = rng.uniform(4, 12, npv)
    data = dict(time=time, lcids=np.repeat(np.arange(nlc), per), pbids=np.arange(nlc) % npb,
                nsamples=1 + np.arange(nlc) % 4, exptimes=0.005 * (np.arange(nlc) % 3), epids=np.arange(nlc) % 3)
    args = (rng.uniform(0.05, 0.2, (npv, npb)), rng.uniform(0.1, 0.4, (npv, npb, 2)),
            2459000.0 + rng.normal(0, 1e-3, (npv, 3)), np.array([2.0, 1.0, 0.6, 4.0]), a,
            np.arccos(rng.uniform(0, 0.9, npv) / a), np.zeros(npv), np.zeros(npv))
    both(data, args)


@pytest.mark.parametrize("npv,npt", [(1, 1), (1, 31), (1, 33), (2, 129), (40, 20000), (600, 20000), (1500, 30001)])
def test_work_split(npv, npt):
    """One point; single slots; whole tiles; several groups of 32 tiles a warp."""
    rng = np.random.default_rng(npv)
    a = rng.uniform(4, 12, npv)
    args = (rng.uniform(0.05, 0.2, (npv, 1)), np.tile([0.3, 0.2], (npv, 1, 1)), rng.normal(0, 1e-3, (npv, 1)),
            rng.uniform(0.7, 9, npv), a, np.arccos(rng.uniform(0, 0.9, npv) / a), np.zeros(npv), np.zeros(npv))
    t = np.linspace(-0.05, 0.05, npt) if npt < 1000 else np.arange(npt) * (2 / 1440)
    both(dict(time=t), args)
