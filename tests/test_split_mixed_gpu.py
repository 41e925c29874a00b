"""Light curves of different sample counts in one data set, in the split path:
tiles of one light curve with one sample per point beside supersampled ones, and
tiles of several (points interleaved, light curves shorter than a tile) whose
counts differ.  Against the FP64 path, with the split path's 1e-6; float64 rows
written by the GPU hold the float32 results' bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["blocks", "interleaved", "short"])
@pytest.mark.parametrize("counts", [(1, 10, 1, 1), (10, 1, 3, 40), (1, 1, 1, 2), (5, 5, 5, 5)])
@pytest.mark.parametrize("npv", [2, 300])
def test_against_fp64(layout, counts, npv):
    from pytransit_gb300 import RoadRunnerModel
    import torch
    rng = np.random.default_rng(npv)
    nlc, npt = 4, 4 * 1100 + 37
    lcids = {"blocks": np.minimum(np.arange(npt) // 1100, 3), "interleaved": np.arange(npt) % 4,
             "short": (np.arange(npt) // 45) % 4}[layout]
    time = 2459000.0 + np.arange(npt) * 0.004
    a, p = rng.uniform(3.5, 12, npv), rng.uniform(0.6, 4, npv)
    p[0], a[0] = 0.25, 1.3                       # every point through the exact fold
    if npv > 4:
        a[2] = 0.9                               # invalid
    counts = np.array(counts)
    args = (rng.uniform(0.05, 0.15, (npv, 2)), rng.uniform(0.1, 0.4, (npv, 2, 2)),
            2459000.0 + rng.normal(0, 1e-3, (npv, 1)), p, a,
            np.arccos(np.minimum(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0), 1.0)), rng.uniform(0, 0.2, npv),
            rng.uniform(0, 6, npv))
    out = {}
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel('quadratic', precision=precision)
        m.set_data(time, lcids=lcids, pbids=np.arange(nlc) % 2, nsamples=counts, exptimes=np.where(counts > 1, 0.02, 0.0))
        out[precision] = m.evaluate(*args, copy=False).double().reshape(npv, -1)
    got, want = out['split'], out['fp64']
    assert torch.equal(got.isnan(), want.isnan())
    assert (got - want).abs().nan_to_num().max().item() <= 1e-6
    rows = torch.full((npv, npt), -7.0, dtype=torch.float64, pin_memory=True)
    m.evaluate(*args, out=rows)
    assert torch.equal(rows.nan_to_num(9.0), got.cpu().nan_to_num(9.0))
