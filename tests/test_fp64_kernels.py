"""FP64 kernel values on the GPU (distance, phase and damping) against sums in
extended precision, at the ends of their ranges: long phases, damping down to
underflow and growth, zero and subnormal distances.
"""
import numpy as np
import pytest

import ifgf_b200 as G
from ifgf_b200 import workloads as W

EPS = 2.0 ** -53
PI = np.longdouble("3.14159265358979323846264338327950288")


def _direct(x, w, k):
    """sum_s w_s e^{k d} / (4 pi d) in extended precision, with the sums of moduli."""
    x = x.astype(np.longdouble)
    d = np.sqrt(((x[:, :, None] - x[:, None, :]) ** 2).sum(0))
    inv = np.where(d > 0, 1 / np.where(d > 0, d, 1), 0) / (4 * PI)
    m = np.exp(np.longdouble(k.real) * d) * inv
    g = m * np.cos(np.longdouble(k.imag) * d) + 1j * (m * np.sin(np.longdouble(k.imag) * d))
    return g @ w, np.abs(g) @ np.abs(w), d.max()


@pytest.mark.gpu
@pytest.mark.parametrize("k", [0.0, 16.0, 150.0])
@pytest.mark.parametrize("scale", [1e-3, 1.0])
def test_oscillating(k, scale):
    x = W.sphere_points(300, seed=3) * scale
    w = W.densities(300, seed=4)
    op = G.HelmholtzIfgfOperator(k, 50, 8)
    op.init(x, x)
    ref, mod, dmax = _direct(x, w, 1j * k)
    # each term: a few roundings of its modulus, k times the distance's rounding
    tol = EPS * (8 + 300 + 2 * k * float(dmax))
    assert np.all(np.abs(op.direct_eval(w, np.arange(300)) - ref) <= tol * mod)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [complex(2.0, -30.0), complex(400.0, 10.0), complex(-40.0, 3.0)])
def test_damped_and_growing(k):
    x = W.sphere_points(300, seed=5)
    w = W.densities(300, seed=6)
    op = G.ModifiedHelmholtzIfgfOperator(k, 50, 8)
    op.init(x, x)
    ref, mod, dmax = _direct(x, w, -k)
    tol = EPS * (8 + 300 + 4 * abs(k) * float(dmax))
    assert np.all(np.abs(op.direct_eval(w, np.arange(300)) - ref) <= tol * mod)


@pytest.mark.gpu
def test_zero_and_subnormal_distances():
    x = W.sphere_points(200, seed=7)
    x[:, 0] = 0.0
    x[:, 1] = (1e-160, 0.0, 0.0)  # squared distance to point 0 below the normal range
    x[:, 2] = x[:, 3]             # coincident: no contribution
    w = W.densities(200, complex_=False, seed=8)
    op = G.LaplaceIfgfOperator(50, 8)
    op.init(x, x)
    ref, mod, _ = _direct(x, w, 0j)
    u = op.direct_eval(w, np.arange(200))
    u_near = op.mult(w)
    assert np.all(np.isfinite(u))
    assert np.all(np.abs(u[2:] - ref.real[2:]) <= EPS * 308 * mod[2:])
    # the square 1e-320 is a subnormal number of 2024 units
    assert np.all(np.abs(u[:2] / ref.real[:2] - 1) <= 1 / 2024)
    assert np.all(np.abs(u_near[:2] / u[:2] - 1) <= 1e-14)
