"""The kernels that prepare a call run beside each other: a captured graph of the
likelihood and its gradient replays to the same bits as the direct calls, on
inputs written between the replays.  And the place of a radius ratio in the
weight table, found without divisions: ratios on the table's rows, between
them, at both ends and outside, against the FP64 path (divisions) to the split
path's 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ['fp64', 'split'])
@pytest.mark.parametrize("npv,ns", [(1, 1), (5, 3), (700, 2)])
def test_captured_likelihood(precision, npv, ns):
    import torch
    from pytransit_gb300 import RoadRunnerModel
    from pytransit_gb300.lnlike import LogLikelihood
    rng = np.random.default_rng(npv)
    m = RoadRunnerModel('quadratic', precision=precision)
    m.set_data(np.linspace(-0.15, 0.15, 400), nsamples=[ns], exptimes=[0.01 if ns > 1 else 0.0])
    dev = lambda x: torch.as_tensor(x, dtype=torch.float64, device='cuda')
    obs = dev(1 + rng.normal(0, 1e-3, 400))

    def draw():
        a = rng.uniform(5, 12, npv)
        return [dev(x) for x in (rng.uniform(0.05, 0.15, (npv, 1)), rng.normal(0, 1e-3, (npv, 1)), np.full(npv, 3.0), a,
                                 np.arccos(rng.uniform(0, 0.8, npv) / a), rng.uniform(0, 0.2, npv),
                                 rng.uniform(0, 6, npv), rng.uniform(0.1, 0.4, (npv, 1, 2)))]

    def run(x):
        lnl = LogLikelihood.apply(m, obs, 1e-3, *x)
        return [lnl.detach(), *torch.autograd.grad(lnl.sum(), x)]

    x = [v.requires_grad_() for v in draw()]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        run(x)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(x)
    for _ in range(3):
        new = draw()
        with torch.no_grad():
            for a, b in zip(x, new):
                a.copy_(b)
        graph.replay()
        got = [o.clone() for o in out]
        assert all(torch.equal(a, b) for a, b in zip(got, run([v.requires_grad_() for v in new])))


@pytest.mark.parametrize("law", ['power-2', 'quadratic'])
def test_place_in_the_table(law):
    from pytransit_gb300 import RoadRunnerModel
    kw = dict(nk=64, klims=(0.05, 0.2))
    rows = np.linspace(0.05, 0.2, 64)
    k = np.concatenate([rows, np.nextafter(rows, 0), np.nextafter(rows, 1), rows[:-1] + np.diff(rows) / 3, [0.02, 0.25]])
    npv = k.size
    out = []
    for precision in ('fp64', 'split'):
        m = RoadRunnerModel(law, precision=precision, **kw)
        m.set_data(np.linspace(-0.1, 0.1, 200))
        out.append(m.evaluate(k[:, None], np.full((npv, 1, 2), 0.4), np.zeros(npv), np.full(npv, 3.0), np.full(npv, 8.0),
                              np.full(npv, 1.5), np.zeros(npv), np.zeros(npv)).reshape(npv, -1))
    assert np.abs(out[0] - out[1]).max() <= 1e-6
