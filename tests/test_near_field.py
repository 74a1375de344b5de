"""FP64 near field at the edges of its staging: boxes of one to hundreds of
points, more near boxes than a CTA's threads, leaves larger than a CTA, one
target, self pairs -- against the FP64 direct sum.  All far pairs are dropped
by the cutoff, so the matvec is the near sum alone where the direct sum is
restricted to the near lists."""
import numpy as np
import pytest

from ifgf_b200 import workloads as W

from .helpers import densities_for, make_gpu_op, rel2


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["helmholtz", "laplace", "combined_field"])
@pytest.mark.parametrize("leaf,n,m", [(400, 700, 700), (1000, 600, 1), (3, 500, 300), (64, 257, 513)])
def test_near_only(name, leaf, n, m):
    src = W.sphere_points(n, seed=0)
    tgt = src if n == m else 0.98 * W.sphere_points(m, seed=1)
    w = densities_for(name, n)
    g = make_gpu_op(name, leaf=leaf, order=8)
    extra = (src,) if name == "combined_field" else ()
    g.init(src, tgt, *extra, cutOff=lambda d: True)  # drop every far pair
    u = g.mult(w)
    pt, ps = g.permutation(1), g.permutation(0)
    # the near lists: source box -> target ranges, in Morton order
    near = np.zeros((m, n), dtype=bool)
    for lev in range(g.levels()):
        ints, _ = g.boxes(lev)
        for b in range(len(ints)):
            for t0, t1 in g.interaction_list(lev, b, far=False):
                near[np.ix_(pt[t0:t1], ps[ints[b, 0]:ints[b, 1]])] = True
    d = src[:, None, :] - tgt[:, :, None]
    r = np.sqrt((d ** 2).sum(0))
    inv = np.where(r > 0, 1 / np.where(r > 0, r, 1), 0)
    if name == "laplace":
        k = inv
    else:
        k = np.exp(20j * r) * inv
        if name == "combined_field":
            nxy = -(d * src[:, None, :]).sum(0)
            k = k * inv * (nxy * inv - 20j * (nxy + r) * (r > 0))
    ref = (np.where(near, k, 0) @ w) / (4 * np.pi)
    assert near.any()
    # a few hundred terms of a few roundings each
    assert rel2(u, ref) <= 1e-12, rel2(u, ref)
