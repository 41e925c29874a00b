"""The split transmission-spectroscopy prologue takes the mean radius ratio from
the FP64 ratios, not from their FP32 values: two sets of ratios with the same
mean (exactly, in FP64) and the same largest one, whose FP32 values have another
mean, give a channel with the same ratio and limb darkening the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npb", [10, 34, 130, 202])
def test_same_mean_same_bits(npb):
    from pytransit_gb300 import TSModel
    rng = np.random.default_rng(npb)
    npv, pairs = 40, npb - 2
    ulp = 2.0 ** -27                                      # FP32's of 0.06 to 0.125
    f = np.round(rng.uniform(0.095, 0.105, (npv, 1)) / ulp) * ulp
    x = f + 0.3125 * ulp
    same = np.tile(x, (1, npb))
    spread = same.copy()
    spread[:, 2:2 + pairs // 2 * 2:2] += 0.3125 * ulp      # FP32: one ulp up
    spread[:, 3:3 + pairs // 2 * 2:2] -= 0.3125 * ulp      # FP32: f, as the others
    same[:, 1] = spread[:, 1] = f[:, 0] + 0.01             # the largest
    assert (spread.astype(np.float32) != same.astype(np.float32)).any()
    np.testing.assert_array_equal(same.sum(1), spread.sum(1))
    a = rng.uniform(5, 12, npv)
    rest = (rng.uniform(0.1, 0.4, (npv, npb, 2)), np.zeros(npv), np.full(npv, 3.0), a,
            np.arccos(rng.uniform(0, 0.8, npv) / a), np.zeros(npv), np.zeros(npv))
    m = TSModel('quadratic', precision='split')
    m.set_data(np.linspace(-0.12, 0.12, 400))
    one = m.evaluate(same, *rest, copy=False)[:, 0].cpu().numpy()
    two = m.evaluate(spread, *rest, copy=False)[:, 0].cpu().numpy()
    assert (one < 1).any(1).all()
    np.testing.assert_array_equal(one, two)
