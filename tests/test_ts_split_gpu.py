"""The split transmission-spectroscopy path where its kernels change form: one
and several chunks of LD-table rows (16 each) and of channels (128), radial
grids of every remainder, points whose samples touch two, three to eight and
more table rows, odd channel counts (channels go in pairs), partial tiles and
unaligned rows, radius ratios in the limb and beyond the star, an invalid
vector and one with a NaN radius ratio.

Against the FP64 path, to the split path's 1e-6; NaN rows match.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law", ['quadratic', 'power-2', 'nonlinear'])
@pytest.mark.parametrize("npv,npb,npt,ns,ex,k0,ng,nzlimb", [
    (1, 1, 1, 1, 0.0, 0.1, 100, 20), (2, 3, 130, 2, 0.001, 0.1, 16, 21), (3, 130, 131, 5, 0.0014, 0.1, 17, 22),
    (5, 7, 1203, 5, 0.003, 0.12, 100, 20), (3, 33, 260, 10, 0.004, 0.1, 100, 23), (2, 257, 515, 5, 0.02, 0.1, 33, 44),
    (4, 5, 400, 3, 0.002, 0.5, 100, 20), (3, 2, 301, 33, 0.03, 0.1, 230, 20), (2, 9, 128, 1, 0.0, 0.15, 48, 20)])
def test_against_fp64(law, npv, npb, npt, ns, ex, k0, ng, nzlimb):
    from pytransit_gb300 import TSModel
    rng = np.random.default_rng(npb + ns)
    ldc = {'quadratic': rng.uniform(0.1, 0.4, (npv, npb, 2)), 'power-2': rng.uniform(0.3, 0.9, (npv, npb, 2)),
           'nonlinear': np.array([0.5, -0.2, 0.6, -0.25]) * rng.uniform(0.8, 1.2, (npv, npb, 4))}[law]
    a = rng.uniform(4, 12, npv)
    k = k0 * rng.uniform(0.95, 1.05, (npv, npb))
    if npv > 2:
        a[1] = 0.7
        k[2, 0] = np.nan
    args = (k, ldc, rng.normal(0, 1e-3, npv), rng.uniform(2, 5, npv), a,
            np.arccos(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0)), rng.uniform(0, 0.2, npv), rng.uniform(0, 6, npv))
    out = []
    for precision in ('fp64', 'split'):
        m = TSModel(law, precision=precision, ng=ng, nzlimb=nzlimb)
        m.set_data(np.linspace(-0.15, 0.15, npt) if npt > 1 else np.array([0.01]), nsamples=[ns], exptimes=[ex])
        out.append(m.evaluate(*args, copy=False).double().cpu().numpy())
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    assert np.nan_to_num(np.abs(out[0] - out[1])).max() <= 1e-6
