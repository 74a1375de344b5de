"""Single FP64 kernel values on the GPU (one source, one target each) against
extended precision, in units of the rounding error, over the range of distances:
from direct_eval, which takes any square of the distance, and from the matvec's
near field, whose loop has seen that the squares are normal numbers."""
import numpy as np
import pytest

import ifgf_b200 as G
from ifgf_b200 import workloads as W

from .helpers import KERNELS, densities_for, make_gpu_op

U = 2.0 ** -53
PI = np.longdouble("3.14159265358979323846264338327950288")


def _values(op, y):
    """(direct_eval, matvec) at the targets y for a source of density 1 at 0; eight
    sources of density 0 around it make every target a near one."""
    r = 0.6 * np.abs(y).max()
    op.init(np.array([(0, 0, 0)] + [(a, b, c) for a in (-r, r) for b in (-r, r) for c in (-r, r)]).T, y)
    w = np.zeros(9, dtype=np.float64 if isinstance(op, G.LaplaceIfgfOperator) else np.complex128)
    w[0] = 1.0
    return op.direct_eval(w, np.arange(y.shape[1])), op.mult(w)


def _targets(m, seed):
    y = W.sphere_points(m, seed=seed)
    return y / np.linalg.norm(y, axis=0) * np.random.default_rng(seed).uniform(0.5, 2.0, m)


def _distance(y):
    return np.sqrt((y.astype(np.longdouble) ** 2).sum(0))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-150, 1e-77, 1.0, 3e77, 1e150])
def test_reciprocal_distance(scale):
    y = _targets(4000, seed=1) * scale
    ref = 1 / (4 * PI * _distance(y))
    # three products and two sums of the square (half of 3 u), the reciprocal
    # root to one unit in the last place (2 u), 1 / (4 pi) and its product (2 u)
    for u in _values(G.LaplaceIfgfOperator(5000, 8), y):
        assert np.max(np.abs(u / ref - 1)) <= 5.5 * U, float(np.max(np.abs(u / ref - 1)) / U)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("kd", [1.0, 60.0, 150.0])
def test_phase(scale, kd):
    y = _targets(4000, seed=2) * scale
    d = _distance(y)
    k = kd / scale
    ph = np.longdouble(k) * d
    ref = (np.cos(ph) + 1j * np.sin(ph)) / (4 * PI * d)
    # the modulus as above; sine and cosine to 3 u; the phase carries k times
    # the distance's error (1.5 u of its square, 1 u of the root)
    tol = U * (5.5 + 3 + 2.5 * ph.astype(np.float64))
    for u in _values(G.HelmholtzIfgfOperator(k, 5000, 8), y):
        assert np.all(np.abs(u / ref - 1) <= tol), float(np.max(np.abs(u / ref - 1) / tol))


@pytest.mark.gpu
@pytest.mark.parametrize("kr", [0.5, 30.0, 300.0, -150.0])
def test_damping(kr):
    y = _targets(4000, seed=3)
    d = _distance(y)
    ref = np.exp(-np.longdouble(kr) * d) / (4 * PI * d)
    tol = U * (5.5 + 3 + 2.5 * abs(kr) * d.astype(np.float64))
    for u in _values(G.ModifiedHelmholtzIfgfOperator(complex(kr, 0.0), 5000, 8), y):
        assert np.all(np.abs(u / ref - 1) <= tol), float(np.max(np.abs(u / ref - 1) / tol))


@pytest.mark.gpu
def test_squares_beyond_the_range():
    """A square that overflows is an infinite distance: no contribution."""
    y = _targets(4000, seed=4) * 1e154
    with np.errstate(over="ignore"):
        d2 = (y ** 2).sum(0)
    ref = np.where(np.isfinite(d2), 1 / (4 * PI * _distance(y)), 0)
    assert (ref == 0).any() and (ref > 0).any()
    for u in _values(G.LaplaceIfgfOperator(5000, 8), y):
        assert np.all(np.abs(u - ref) <= 5.5 * U * ref)


@pytest.mark.gpu
def test_damping_to_underflow():
    """Values from e^{-200} down through the subnormal numbers to zero."""
    y = _targets(4000, seed=5)
    d = _distance(y)
    ref = np.exp(-np.longdouble(400) * d) / (4 * PI * d)
    tiny = np.longdouble(2) ** -1074
    assert (ref > 2 ** -1000).any() and ((ref < 2 ** -1023) & (ref > 8 * tiny)).any()
    # as test_damping, and up to four roundings to whole subnormal units
    tol = U * (5.5 + 3 + 2.5 * 400 * d) * ref + 2 * tiny
    for u in _values(G.ModifiedHelmholtzIfgfOperator(400 + 0j, 5000, 8), y):
        assert np.all(np.abs(u - ref) <= tol), float(np.max(np.abs(u - ref) / tol))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["modified_helmholtz", "grad_helmholtz", "double_layer"])
def test_leaf_with_steep_damping(name):
    """Damping across a leaf of more than the normal range's octaves: the far
    values underflow and stay finite on the way."""
    src = W.sphere_points(300, seed=6)
    op = make_gpu_op(name, leaf=500, order=8, dx=0, k=complex(380.0, 3.0))
    tgt = 0.3 * W.sphere_points(200, seed=7) + np.array([[5.0], [0.0], [0.0]])
    op.init(src, tgt, *((src,) if KERNELS[name][2] else ()))
    assert op.stats()["target_leaf_far_evals"] > 0
    assert np.all(op.mult(densities_for(name, 300)) == 0)
