"""The fused FP64 prologue (rr_prepare_f64_ld) against the two stages it
replaces (rr_ld_tables_f64, then rr_prepare_f64), through the C ABI: istar
bit for bit, and the flux from the two workspaces to 1e-14 (a LD mean differs
by the rounding of a few sums of order one, ~1e-15, and enters the flux times
the overlap area over istar, below 0.4).  Every law the fused kernel takes and
two that it hands on, radius ratios outside the weight table, one per
passband, invalid orbits and a NaN coefficient.
"""
import numpy as np
import pytest

from test_prologue_gpu import LAWS, _coefs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("law,npar", LAWS)
@pytest.mark.parametrize("npv,npb,ecc", [(1, 1, 0.0), (33, 3, 0.3), (131, 50, 0.3)])
def test_fused_prologue_matches_two_stages(law, npar, npv, npb, ecc):
    import torch
    from pytransit_gb300 import RoadRunnerModel, _lib
    rng = np.random.default_rng(npv)
    m = RoadRunnerModel(law)
    m.set_data(np.tile(np.linspace(-0.2, 0.2, 150), npb), lcids=np.repeat(np.arange(npb), 150), pbids=np.arange(npb))
    k = rng.uniform(0.05, 0.15, (npv, npb))
    k[::31, 0] = 0.6
    a = rng.uniform(3, 20, npv)
    a[npv // 2] = 0.9 if npv > 1 else 5.0
    ldc = _coefs(law, rng, (npv, npb))
    if npar and npv > 1:
        ldc[5, 0, 0] = np.nan
    prm = dict(k=k, t0=rng.normal(0, 1e-3, (npv, 1)), p=rng.uniform(1, 5, npv), a=a,
               i=np.arccos(rng.uniform(0, 0.9, npv) / np.maximum(a, 1.0)), e=rng.uniform(0, ecc, npv),
               w=rng.uniform(0, 6, npv), ldc=ldc)
    dev = torch.device("cuda")
    d = {n: torch.as_tensor(np.ascontiguousarray(v)).to(dev) for n, v in prm.items()}
    dd, tb = m._device_data(dev), m._device_tables(dev)
    L, P, sp = _lib.lib(), _lib.ptr, _lib.stream_ptr(dev)
    nz, ng, nk, npt = m.ze.size, m.ng, m.nk, m.npt
    basis, nb = m._basis(dev, npar, False)
    kmin, kmax = float(m.klims[0]), float(m.klims[1])
    wsb = L.rr_full_f64_workspace_bytes(npv, npb, ng)
    orbit = (P(d["k"]), npb, P(d["p"]), P(d["a"]), P(d["i"]), P(d["e"]), P(d["w"]), npv, npb)
    res = []
    for fused in (True, False):
        ldp = torch.empty((npv, npb, nz), dtype=torch.float64, device=dev)
        ist = torch.empty((npv, npb), dtype=torch.float64, device=dev)
        ws = torch.empty(wsb, dtype=torch.uint8, device=dev)
        f = torch.empty((npv, npt), dtype=torch.float64, device=dev)
        if fused:
            _lib.check(L.rr_prepare_f64_ld(*orbit, m.ld_law, P(d["ldc"]), npar, P(tb["mu"]), nz, P(basis), nb,
                                           P(tb["W64"]), nk, ng, m.dk, kmin, kmax, P(tb["ze"]), P(ldp), P(ist),
                                           P(ws), wsb, sp))
        else:
            _lib.check(L.rr_ld_tables_f64(m.ld_law, P(d["ldc"]), npv, npb, npar, P(tb["mu"]), nz, P(ldp), P(ist),
                                          sp))
            _lib.check(L.rr_prepare_f64(*orbit, P(ldp), P(tb["W64"]), nk, ng, nz, m.dk, kmin, kmax, P(tb["ze"]),
                                        P(ws), wsb, sp, m.ld_law, P(d["ldc"]), npar, P(basis), nb))
        _lib.check(L.rr_flux_f64(P(dd["time"]), npt, P(d["k"]), npb, P(d["t0"]), 1, P(d["p"]), npv, npb, npb,
                                 P(dd["lcids"]), P(dd["pbids"]), P(dd["epids"]), P(dd["nsamples"]),
                                 P(dd["exptimes"]), P(ist), ng, m.dg, P(ws), P(f), npt, sp))
        res.append((ist.cpu().numpy(), f.cpu().numpy()))
    (i1, f1), (i2, f2) = res
    np.testing.assert_array_equal(i1, i2)
    assert np.array_equal(np.isnan(f1), np.isnan(f2))
    if npv > 1:
        assert np.isnan(f1[npv // 2]).all() and (not npar or np.isnan(f1[5]).all())
    assert (f1 < 1.0).any() and np.nanmax(np.abs(f1 - f2)) <= 1e-14
