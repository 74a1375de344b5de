"""Orders 11 and 12 (fixed-order kernels) and 7 (runtime orders) against the
oracle in FP64 and, at the high orders, mixed within FP32 rounding of FP64."""
import numpy as np
import pytest

from ifgf_b200 import workloads as W

from .helpers import densities_for, init_op, make_gpu_op, make_oracle_op, rel2


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["helmholtz", "laplace", "modified_helmholtz", "double_layer"])
@pytest.mark.parametrize("order", [7, 11, 12])
def test_parity(name, order):
    n = 2503
    pts = W.ellipsoid_points(n, seed=0)
    w = densities_for(name, n)
    g = make_gpu_op(name, leaf=40, order=order)
    o = make_oracle_op(name, leaf=40, order=order)
    init_op(g, name, pts, pts)
    init_op(o, name, pts, pts)
    u, uo = g.mult(w), o.mult(w)
    assert rel2(u, uo) <= 1e-12, rel2(u, uo)
    g.set_far_plan(False)
    assert rel2(g.mult(w), uo) <= 1e-12
    assert g.stats()["missing_cone_lookups"] == 0
    if order == 7:
        return
    g.set_precision("mixed")
    # the mixed pipeline's tolerance against FP64
    assert rel2(g.mult(w), uo) <= 2e-5, rel2(g.mult(w), uo)
    assert rel2(g.mult_batch(np.stack([w, w]))[1], uo) <= 2e-5
