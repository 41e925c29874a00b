"""A log-likelihood workspace for a population serves every smaller one and every
shorter row."""
import numpy as np
import pytest


@pytest.mark.parametrize("split", [0, 1])
def test_workspace_does_not_shrink(split):
    from pytransit_gb300 import _lib
    import pytransit_gb300.lnlike  # noqa: F401  (declares the entry point)
    L = _lib.lib()

    def size(npv, npt):
        return L.rr_lnlike_workspace_bytes(split, npv, 1, 1, 1, 100, 2, npt, 1)
    for npt in (1, 128, 1000, 3000, 19700):
        s = [size(n, npt) for n in range(1, 2001)]
        assert all(a <= b for a, b in zip(s, s[1:]))
    for npv in (1, 25, 26, 203, 1500):
        s = [size(npv, n) for n in range(1, 20001, 37)]
        assert all(a <= b for a, b in zip(s, s[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("npt,pairs", [(3000, [(26, 25), (51, 50), (203, 202), (304, 303), (406, 405)]),
                                       (20000, [(32, 31), (1500, 63), (2000, 1)])])
def test_smaller_call_in_a_larger_calls_workspace(npt, pairs):
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import lnlikelihood
    rng = np.random.default_rng(npt)
    npv = max(max(p) for p in pairs)
    time = np.linspace(-0.2, 0.2, npt) if npt < 5000 else np.arange(npt) * (2 / 1440)
    a = rng.uniform(6, 12, npv)
    prm = [rng.uniform(0.08, 0.12, (npv, 1)), rng.uniform(0.1, 0.4, (npv, 1, 2)), rng.normal(0, 1e-3, (npv, 1)),
           np.full(npv, 3.0), a, np.arccos(rng.uniform(0.1, 0.8, npv) / a), rng.uniform(0.05, 0.2, npv),
           rng.uniform(0, 6, npv)]
    obs = 1.0 + rng.normal(0, 1e-3, npt)
    for large, small in pairs:
        m = RoadRunnerModel('quadratic')
        m.set_data(time)
        lnl, g = lnlikelihood(m, obs, 1e-3, *(v[:large] for v in prm), grad=True)
        ws = m._ws
        lnl2, g2 = lnlikelihood(m, obs, 1e-3, *(v[:small] for v in prm), grad=True)
        assert m._ws is ws                       # nothing larger was asked for
        np.testing.assert_allclose(lnl2, lnl[:small], rtol=1e-12)     # sums of terms of one sign, in another order
        assert (np.abs(g2 - g[:small]).max(0) <= 1e-10 * np.abs(g).max(0)).all()
