"""The split flux kernel's supersampled path at the sizes where it changes
form: sample counts below, at and above the rows evaluated at once, light
curves shorter than a tile (tiles of many of them), partial tiles, radius
ratios on both sides of the limb forms' ranges, launches of one and of many
tiles per warp, a window that fills the period.  Against the FP64 path, with
the split path's 1e-6; float64 rows hold the float32 results' bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [2, 3, 5, 9, 10, 11, 40])
@pytest.mark.parametrize("npv,nlc,per,k0", [(1, 1, 1, 0.1), (2, 1, 129, 0.1), (3, 30, 17, 0.2), (40, 3, 4001, 0.1),
                                            (5, 2, 300, 0.6), (3, 1, 260, 1.2)])
def test_against_fp64(ns, npv, nlc, per, k0):
    import torch
    from pytransit_gb300 import RoadRunnerModel
    rng = np.random.default_rng(ns * per)
    a = rng.uniform(3.5, 12, npv)
    p = rng.uniform(0.6, 4, npv)
    if npv > 4:
        p[3], a[3] = 0.25, 1.3                  # every point through the exact fold
        a[2] = 0.9                              # invalid
    step = 0.004 if per < 1000 else 0.02
    time = np.concatenate([2459000.0 + 0.5 * j - 0.3 + np.arange(per) * step for j in range(nlc)])
    counts = np.full(nlc, ns)
    counts[-1] = 1 if nlc > 1 else ns           # single-sample light curves beside supersampled ones
    data = dict(time=time, lcids=np.repeat(np.arange(nlc), per), pbids=np.arange(nlc) % 2 if nlc > 1 else [0],
                nsamples=counts, exptimes=np.where(counts > 1, 0.02, 0.0))
    npb = min(nlc, 2)
    args = (k0 * rng.uniform(0.9, 1.1, (npv, npb)), rng.uniform(0.1, 0.4, (npv, npb, 2)),
            2459000.0 + rng.normal(0, 1e-3, (npv, 1)), p, a,
            np.arccos(np.minimum(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0), 1.0)), rng.uniform(0, 0.2, npv),
            rng.uniform(0, 6, npv))
    out = {}
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel('quadratic', precision=precision)
        m.set_data(**data)
        out[precision] = m.evaluate(*args, copy=False).double().reshape(npv, -1)
    got, want = out['split'], out['fp64']
    assert torch.equal(got.isnan(), want.isnan())
    assert (got - want).abs().nan_to_num().max().item() <= 1e-6
    rows = torch.full((npv, time.size), -7.0, dtype=torch.float64, pin_memory=True)
    m.evaluate(*args, out=rows)
    assert torch.equal(rows.nan_to_num(9.0), got.cpu().nan_to_num(9.0))
