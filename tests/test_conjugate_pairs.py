"""Multi-wavenumber batches with conjugate pairs in any order: the planes of a
pair share their kernel values; every row equals the batch of its wavenumber
alone (FP32 sums of the same terms: 1e-6)."""
import numpy as np
import pytest

from ifgf_b200 import workloads as W

from .helpers import densities_for, init_op, make_gpu_op, rel2

# small, so that all give the operator's cone grids
Z = 0.1 * np.array([0.5 + 3j, 2.0 + 1j, 1.5, 0.5 - 3j, 3 - 2j, 2.0 - 1j, 1.5, 0.25 + 2j, 2.0 - 1j])
CONTOUR = 0.3 * (1 - 0.45 * np.exp(2j * np.pi * np.arange(10) / 10))  # conjugate to rounding


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["modified_helmholtz", "grad_helmholtz", "double_layer"])
@pytest.mark.parametrize("ks", [Z, Z[:1], CONTOUR], ids=["mixed", "one", "contour"])
def test_pairs_equal_single_planes(name, ks):
    n = 3001
    pts = W.sphere_points(n, seed=0)
    g = make_gpu_op(name, leaf=40, order=8, dx=1, k=0.2 + 0.1j)
    init_op(g, name, pts, pts)
    g.set_precision("mixed")
    w = np.stack([densities_for(name, n, seed=5 + i) for i in range(len(ks))])
    u = g.mult_wavenumbers(ks, w)
    assert g.stats()["missing_cone_lookups"] == 0
    for i, k in enumerate(ks):
        one = g.mult_wavenumbers([k], w[i:i + 1])[0]
        assert rel2(u[i], one) <= 1e-6, (i, rel2(u[i], one))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["modified_helmholtz", "grad_helmholtz", "helmholtz"])
def test_more_wavenumbers_than_one_launch_takes(name):
    """73 wavenumbers (a launch takes 64): pairs that end up on both sides of
    the cut, singles, shuffled; host and device entry points, row by row."""
    import torch

    n, rng = 1501, np.random.default_rng(3)
    z = rng.uniform(0.1, 0.3, 33) + 1j * rng.uniform(0.05, 0.3, 33)
    ks = np.concatenate([z, z.conj(), rng.uniform(0.1, 0.3, 7) + 0.31j])
    if name == "helmholtz":
        ks = np.abs(ks).astype(complex)
    ks = ks[rng.permutation(len(ks))]
    pts = W.sphere_points(n, seed=0)
    g = make_gpu_op(name, leaf=40, order=8, dx=1, k=0.2 if name == "helmholtz" else 0.2 + 0.1j)
    init_op(g, name, pts, pts)
    g.set_precision("mixed")
    w = np.stack([densities_for(name, n, seed=5 + i) for i in range(len(ks))])
    u = g.mult_wavenumbers(ks, w)
    dw = torch.from_numpy(w).cuda()
    du = torch.empty_like(dw)
    g.mult_wavenumbers_device(ks, dw.data_ptr(), du.data_ptr())
    assert np.array_equal(du.cpu().numpy(), u)
    for i, k in enumerate(ks):
        one = g.mult_wavenumbers([k], w[i:i + 1])[0]
        assert rel2(u[i], one) <= 1e-6, (i, rel2(u[i], one))
