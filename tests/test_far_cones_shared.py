"""Far-cone plans beside other users of the device: another thread's stream
capture, memory that others need."""
import threading

import numpy as np
import pytest

from ifgf_b200 import IfgfError
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


def _free():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _hold_all_but(n_bytes):
    """A tensor that leaves about n_bytes of the device's memory."""
    import torch

    return torch.empty(_free() - n_bytes, dtype=torch.uint8, device="cuda")


def _op(n, pts):
    g = make_gpu_op("helmholtz", leaf=100, order=8)
    g.init(pts, pts)
    g.set_precision("mixed")
    g.set_upward_path("ffma")
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("same", [True, False])
def test_plans_give_way_to_other_allocations(same):
    """A batch whose planes find no room beside a plan -- the operator's own or
    another operator's -- gets the plan's memory; later matvecs go on without or
    build it again."""
    n, rhs = 100000, 4
    pts = W.sphere_points(n, seed=0)
    w = np.stack([W.densities(n, seed=i) for i in range(rhs)])
    a = _op(n, pts)
    b = a if same else _op(n, pts)
    ref = a.mult(w[0])
    plan = a.stats()["far_cones"]["bytes"]
    assert plan > 100 << 20
    # what a batch takes: of an operator of its own
    twin = _op(n, pts)
    before = _free()
    twin.mult_batch(w)
    need = before - _free()
    del twin
    # (the staging buffers of host calls are a few MB of it)
    held = _hold_all_but(need - plan // 2)
    u = b.mult_batch(w)
    assert a.stats()["far_cones"]["bytes"] == 0
    del held
    _free()
    assert rel2(u[0], ref) <= 1e-6
    assert rel2(a.mult(w[0]), ref) <= 1e-6


@pytest.mark.gpu
def test_batch_after_one_that_found_no_memory():
    n = 20000
    pts = W.sphere_points(n, seed=0)
    w = np.stack([W.densities(n, seed=i) for i in range(64)])
    a = _op(n, pts)
    a.set_far_plan(False)
    ref = a.mult_batch(w[:2])
    held = _hold_all_but(64 << 20)
    with pytest.raises(IfgfError, match="out of memory"):
        a.mult_batch(w)
    del held
    _free()
    assert rel2(a.mult_batch(w[:2]), ref) <= 1e-6


@pytest.mark.gpu
def test_plan_refused_for_want_of_memory_is_tried_again():
    import torch

    n = 50000
    pts = W.sphere_points(n, seed=0)
    w = torch.from_numpy(W.densities(n, seed=1)).cuda()
    g = make_gpu_op("helmholtz", leaf=100, order=8)
    g.init(pts, pts)
    us = []

    def mult():
        us.append(torch.empty_like(w))
        g.mult_device(w.data_ptr(), us[-1].data_ptr())
        torch.cuda.synchronize()
        return g.stats()["far_cones"]

    us_room = torch.empty(32, n, dtype=w.dtype, device="cuda")  # for the results
    held = _hold_all_but(64 << 20)
    del us_room
    st = mult()
    assert st["built"] == 0 and st["refused"] == 1
    del held
    _free()
    calls = 0
    while not st["built"]:
        st = mult()
        calls += 1
        assert calls <= 16
    assert st["refused"] == 0
    for u in us[1:]:
        assert rel2(u.cpu().numpy(), us[0].cpu().numpy()) <= 1e-12


@pytest.mark.gpu
def test_mixed_plan_takes_the_unused_reservation():
    n = 4000
    pts = W.sphere_points(n, seed=0)
    w = W.densities(n, seed=1)
    g = make_gpu_op("helmholtz", leaf=50, order=8)
    g.init(pts, pts)
    assert g.stats()["far_cones"]["bytes"] > 0  # with init's buffers
    g.set_precision("mixed")
    um = g.mult(w)
    assert g.stats()["far_cones"]["built"] == 1
    g.set_precision("fp64")
    assert g.stats()["far_cones"]["bytes"] == 0
    u = g.mult(w)
    assert g.stats()["far_cones"]["built"] == 1
    g.set_precision("mixed")
    assert np.array_equal(g.mult(w), um)
    assert rel2(um, u) <= 2e-5
