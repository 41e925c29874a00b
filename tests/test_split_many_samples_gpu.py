"""The error of the split path's supersampled sums does not grow with the number
of samples: a large planet inside the star (a deficit of 0.1 to 0.5, terms of
nearly one size, whose roundings have one sign) with up to 4000 samples a point.

Against the FP64 path.  Tolerance, in u = 2^-24: per sample z, the table position
and the lerp (about 6 u), the area (2 u), the sum as a tree (log2 of 10, 4 u) and a
compensated sum, the products with 1/istar and 1/ns (4 u), all of a deficit below
0.55, and the result's rounding: 0.55 x 16 u + u = 6e-7.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [7, 10, 11, 40, 300, 1000, 4000])
@pytest.mark.parametrize("npt,interleaved", [(160, False), (160, True), (256, False)])   # tiles of one and of two light curves
def test_error_does_not_grow(ns, npt, interleaved):
    from pytransit_gb300 import RoadRunnerModel
    npv = 12
    k = np.linspace(0.3, 0.68, npv).reshape(-1, 1)
    time = np.linspace(-0.004, 0.004, npt)                   # z below 0.1: inside for every k
    args = (k, np.tile([0.3, 0.2], (npv, 2, 1)), 0.0, np.full(npv, 10.0), np.full(npv, 15.0),
            np.full(npv, np.arccos(0.05 / 15)), np.zeros(npv), np.zeros(npv))
    lcids = np.arange(npt) % 2 if interleaved else np.repeat([0, 1], npt // 2)
    out = {}
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel('quadratic', precision=precision)
        m.set_data(time, lcids=lcids, pbids=[0, 1], nsamples=[ns, ns], exptimes=[0.002, 0.002])
        out[precision] = m.evaluate(*args, copy=False).double().cpu().numpy()
    err = np.abs(out['split'] - out['fp64']).max()
    assert err <= 6e-7, err
