"""The far-cone plans of the single matvec (pairs sorted by fine cone) against
the far kernels that look every pair up.  Both evaluate the same interpolants.
FP64 (sums on the FP64 tensor cores): the local coordinates are formed from
other roundings (a few 1e-16, amplified by the degree squared and the cone
count), so the results agree to 1e-12 of their norm, the parity tolerance.
Mixed: the same FP32 coordinates and terms, summed in another order.
"""
import numpy as np
import pytest

from ifgf_b200 import workloads as W

from .helpers import KERNELS, densities_for, init_op, make_gpu_op, rel2

TOL = 1e-12
TOL_MIXED = 1e-6


def _both(op, w):
    u = op.mult(w)
    st = op.stats()["far_cones"]
    again = op.mult(w)
    op.set_far_plan(False)
    assert op.stats()["far_cones"]["built"] == 0
    ref = op.mult(w)
    op.set_far_plan(True)
    assert np.array_equal(u, again)  # fixed order of the sums
    assert op.stats()["missing_cone_lookups"] == 0
    return u, ref, st


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(KERNELS))
@pytest.mark.parametrize("order", [8, 9, 10])
def test_all_kernels_and_orders(name, order):
    n = 4001
    pts = W.sphere_points(n, seed=0)
    g = make_gpu_op(name, leaf=40, order=order)
    init_op(g, name, pts, pts)
    u, ref, st = _both(g, densities_for(name, n))
    assert st["built"] == 1 and st["places"] % 32 == 0 and st["pairs"] > 0
    assert rel2(u, ref) <= TOL, rel2(u, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("leaf,n,m", [(5, 900, 3000), (400, 6000, 20000), (64, 3000, 7)])
def test_other_targets_and_leaf_sizes(leaf, n, m):
    """Targets off the sources, from a few per leaf to leaves of more than a
    CTA's threads; a target above a box's centre (no azimuth)."""
    src = W.sphere_points(n, seed=1)
    tgt = 1.5 * W.ellipsoid_points(m, seed=2)
    g = make_gpu_op("helmholtz", leaf=leaf, order=9)
    g.init(src, tgt)
    ints, bb = g.boxes(min(2, g.levels() - 1))
    tgt[:, 0] = [(bb[0, 0] + bb[0, 3]) / 2, (bb[0, 1] + bb[0, 4]) / 2, 40.0]
    g.init(src, tgt)
    u, ref, _ = _both(g, W.densities(n, seed=3))
    assert np.all(np.isfinite(u))
    assert rel2(u, ref) <= TOL, rel2(u, ref)


@pytest.mark.gpu
def test_sharded_and_k_derivative():
    n = 6000
    pts = W.sphere_points(n, seed=0)
    w = W.densities(n, seed=1)
    g = make_gpu_op("helmholtz", leaf=50, order=8)
    g.init(pts, pts)
    total, dk = g.mult(w), g.mult_dk(w)
    g.set_far_plan(False)
    assert rel2(dk, g.mult_dk(w)) <= TOL
    parts = 0
    for r in range(3):
        s = make_gpu_op("helmholtz", leaf=50, order=8)
        s.set_shard(r, 3)
        s.init(pts, pts)
        parts = parts + s.mult(w)
    assert rel2(parts, total) <= TOL


@pytest.mark.gpu
def test_capture():
    """A first call inside a capture records the lookup kernel; a captured plan
    outlives set_far_plan(False)."""
    import torch

    n = 3000
    pts = W.sphere_points(n, seed=0)
    g = make_gpu_op("helmholtz", leaf=50, order=8)
    g.init(pts, pts)
    w = torch.from_numpy(W.densities(n, seed=1)).cuda()
    u = torch.empty_like(w)
    ref = torch.empty_like(w)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()

    def captured():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            g.mult_device(w.data_ptr(), u.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return graph

    first = captured()
    assert g.stats()["far_cones"]["built"] == 0
    g.mult_device(w.data_ptr(), ref.data_ptr())
    assert g.stats()["far_cones"]["built"] == 1
    second = captured()
    g.set_far_plan(False)
    for graph in (first, second):
        u.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert float((u - ref).norm() / ref.norm()) <= TOL
    del first, second


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(KERNELS))
@pytest.mark.parametrize("order", [8, 9, 10, 12])
def test_mixed(name, order):
    n = 4001
    pts = W.sphere_points(n, seed=0)
    g = make_gpu_op(name, leaf=40, order=order)
    init_op(g, name, pts, pts)
    g.set_precision("mixed")
    g.set_upward_path("ffma")  # the autotuner's choice would be timed again
    u, ref, st = _both(g, densities_for(name, n))
    assert st["built"] == 1
    assert rel2(u, ref) <= TOL_MIXED, rel2(u, ref)


@pytest.mark.gpu
def test_both_precisions_keep_their_plans():
    n = 3000
    pts = W.sphere_points(n, seed=0)
    w = W.densities(n, seed=1)
    g = make_gpu_op("helmholtz", leaf=50, order=8)
    g.init(pts, pts)
    u = g.mult(w)
    g.set_precision("mixed")
    um = g.mult(w)
    assert rel2(um, u) <= 2e-5
    g.set_precision("fp64")
    assert np.array_equal(g.mult(w), u)
