"""Far-cone plans beside other users of the device: another thread's stream
capture, memory that others need."""
import threading

import numpy as np
import pytest

from ifgf_b200 import workloads as W

from .helpers import make_gpu_op, rel2


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_call_while_another_thread_captures(precision):
    """The first matvec of an operator builds its plan on its own stream alone,
    so it neither fails nor ends the capture of a non-blocking stream."""
    import torch

    n = 3000
    pts = W.sphere_points(n, seed=0)
    w = torch.from_numpy(W.densities(n, seed=1)).cuda()
    a, b = make_gpu_op("helmholtz", leaf=50, order=8), make_gpu_op("helmholtz", leaf=50, order=8)
    for op in (a, b):
        op.init(pts, pts)
        op.set_precision(precision)
        op.set_upward_path("ffma")
    ua, ub = torch.empty_like(w), torch.empty_like(w)
    if precision == "mixed":  # its other tables
        a.set_far_plan(False)
        a.mult_device(w.data_ptr(), ua.data_ptr())
        a.set_far_plan(True)
    b.mult_device(w.data_ptr(), ub.data_ptr())
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    errors = []

    def first_call():
        try:
            a.mult_device(w.data_ptr(), ua.data_ptr(), sa.cuda_stream)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=sb):
        t = threading.Thread(target=first_call)
        t.start()
        t.join()
        b.mult_device(w.data_ptr(), ub.data_ptr(), sb.cuda_stream)
    assert not errors, errors
    assert a.stats()["far_cones"]["built"] == 1
    ub.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert rel2(ua.cpu().numpy(), ub.cpu().numpy()) <= 1e-12
    assert np.isfinite(ua.abs().sum().item())
    del graph
