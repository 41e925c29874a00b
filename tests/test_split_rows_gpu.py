"""rr_flux_split_rows: the same values with and without RR_ROWS_TILES for data sets of
every kind (to the split path's 1e-6 where the two take supersampled points
through different sums, the same bits where they do not), and what it refuses."""
import numpy as np
import pytest


def test_refused_without_gpu():
    import ctypes
    from pytransit_gb300 import _lib
    L, dev = _lib.lib(), ctypes.c_void_p(256)

    def rows(pv0, pv1, ld, kind):
        return L.rr_flux_split_rows(dev, 100, dev, 8, 1, 1, 100, 0.01, dev, pv0, pv1, dev, ld, kind, None)
    assert rows(0, 9, 100, 0) == 2 and rows(5, 4, 100, 0) == 2 and rows(0, 8, 99, 0) == 2
    assert rows(0, 8, 100, 8) == 2 and rows(0, 8, 100, -1) == 2       # unknown kinds
    assert rows(3, 3, 100, 7) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("counts,per", [((1, 1, 1), 500), ((10, 10, 10), 500), ((1, 10, 1), 500), ((5, 5, 5), 60)])
def test_kinds_agree(counts, per):
    import torch
    from pytransit_gb300 import RoadRunnerModel, _lib
    rng = np.random.default_rng(per)
    npv, nlc = 50, 3
    npt = per * nlc
    time = 2459000.0 + np.arange(npt) * 0.004
    a = rng.uniform(3.5, 12, npv)
    a[1] = 0.9
    m = RoadRunnerModel('quadratic', precision='split')
    m.set_data(time, lcids=np.repeat(np.arange(nlc), per), pbids=np.zeros(nlc, int), nsamples=counts,
               exptimes=[0.02 if c > 1 else 0.0 for c in counts])
    want = m.evaluate(rng.uniform(0.05, 0.15, (npv, 1)), rng.uniform(0.1, 0.4, (npv, 1, 2)),
                      2459000.0 + rng.normal(0, 1e-3, (npv, 1)), rng.uniform(0.6, 4, npv), a,
                      np.arccos(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0)), np.zeros(npv), np.zeros(npv), copy=False)
    L, P = _lib.lib(), _lib.addr
    dd = m._device_data(want.device)
    assert dd['rows'] == (0 if counts == (10, 10, 10) else _lib.ROWS_TILES)
    same = counts != (10, 10, 10)
    for kind in range(8):
        f64 = kind & _lib.ROWS_F64
        out = torch.ones((npv, npt), dtype=torch.float64 if f64 else torch.float32, device=want.device)
        assert L.rr_flux_split_rows(P(dd['times_ff']), npt, P(dd['lcids']), npv, nlc, 1, m.ng, m.dg, P(m._ws), 0, npv,
                                    P(out), npt, kind, _lib.stream_addr(want.device)) == 0
        torch.cuda.synchronize()
        diff = (out.double() - want.double()).abs()
        assert torch.equal(out.isnan(), want.isnan())
        assert diff.nan_to_num().max().item() <= (0.0 if same or not kind & _lib.ROWS_TILES else 1e-6)
