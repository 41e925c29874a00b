"""Limb-darkening means from a weight table that does not start on a 16-byte
boundary (element-wise staging, rows padded), at the largest radial grid, odd
and even numbers of rows and a full group of passbands, where the profiles end
exactly at the end of their shared memory.  Against the oracle, 1e-9 (FP64) and
1e-6 (split).
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [('fp64', 1e-9), ('split', 1e-6)])
@pytest.mark.parametrize("nzin,nzlimb", [(32, 32), (31, 32)])
@pytest.mark.parametrize("ng", [100, 101])
@pytest.mark.parametrize("k0", [0.1, 0.4])      # inside the table; the 2D table
def test_unaligned_weights(precision, tol, nzin, nzlimb, ng, k0):
    import torch
    from pytransit_gb300 import RoadRunnerModel
    rng = np.random.default_rng(ng)
    npv, npb, per = 3, 4, 80
    kw = dict(nzin=nzin, nzlimb=nzlimb, ng=ng, nk=32, klims=(0.05, 0.2))
    data = dict(time=np.tile(np.linspace(-0.1, 0.09, per), npb), lcids=np.repeat(np.arange(npb), per),
                pbids=np.arange(npb))
    a = rng.uniform(6, 12, npv)
    prm = (k0 * rng.uniform(0.9, 1.1, (npv, npb)), rng.uniform(0.3, 0.8, (npv, npb, 2)), rng.normal(0, 1e-3, npv),
           np.full(npv, 3.0), a, np.arccos(rng.uniform(0.1, 0.6, npv) / a), np.zeros(npv), np.zeros(npv))
    ref = oracle.OracleRoadRunner('power-2', **kw)
    ref.set_data(**data)
    m = RoadRunnerModel('power-2', precision=precision, **kw)
    m.set_data(**data)
    tb = m._device_tables(m._cuda_device())
    name = 'W32' if precision == 'split' else 'W64'
    W = tb[name]
    shifted = torch.empty(W.numel() + 1, dtype=W.dtype, device=W.device)[1:].view(W.shape)
    shifted.copy_(W)
    assert shifted.data_ptr() % 16
    tb[name] = shifted
    got = m.evaluate(*prm).reshape(npv, -1)
    assert np.abs(got - ref.evaluate(*prm).reshape(npv, -1)).max() <= tol
