"""The pinned staging buffer of a model's uploads: a model that is collected, or one
that uploads, while a CUDA graph is being captured does not break the capture."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model():
    from pytransit_gb300 import RoadRunnerModel
    m = RoadRunnerModel('quadratic')
    m.set_data(np.linspace(-0.1, 0.1, 500))
    return m, lambda: m.evaluate(0.1, [[[0.4, 0.2]]], 0.0, 3.0, 8.0, 1.55, 0.0, 0.0, copy=False)


def test_release_during_capture():
    import torch
    m, call = model()
    call()
    x = torch.zeros(8, device='cuda')
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        x += 1
        del m, call
        gc.collect()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()


def test_wait_in_another_thread_during_capture():
    """A thread waits for its staging buffer while this one captures."""
    import torch
    from pytransit_gb300 import _lib
    dev = torch.device('cuda', torch.cuda.current_device())
    st = _lib.Staging(1024, dev)
    st.put(dict(a=np.ones(100)))
    torch.cuda.synchronize()
    status = []
    x = torch.zeros(8, device='cuda')
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        t = threading.Thread(target=lambda: status.append(_lib.lib().rr_event_wait(st._event)))
        t.start()
        t.join()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert status == [0] and (x == 2).all()
