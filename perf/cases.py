"""Measured cases of the IFGF matvec: the calls a program makes once it has an operator.

A case is a dict of plain values:

  kind       kernel plug-in: laplace, helmholtz, modified, gradient, double_layer, combined
  call       host         op.mult on numpy arrays
             device       op.mult_device on CUDA buffers
             batch_host   op.mult_batch on pinned host arrays, into a pinned result
             batch        op.mult_batch_device, several right-hand sides
             wavenumbers  op.mult_wavenumbers_device, one right-hand side per wavenumber
             gradients    autograd: u = A x, then d/dx and d/dk of |u - b|^2 / 2
  n, m       sources on the surface; m targets (0: the targets are the sources)
  surface    sphere (radius 1) or ellipsoid (semi-axes 1, 1, 0.5); with m > 0
             the targets lie on a sphere of radius 1.25 around it
  k_re, k_im wavenumber as the operator takes it (ignored by laplace)
  leaf, order, precision   as the operator takes them
  rhs        right-hand sides (wavenumbers for the call of that name)

Densities are i.i.d. standard normal (real and imaginary part).  A mixed
operator's densities hold 32-bit values and its result, whose sums are in 32
bits, is handed on in complex64 as such a program keeps it; the library's own
buffers are complex128 in either precision.
"""
import math

import numpy as np
import torch

import ifgf_b200 as G
from ifgf_b200 import workloads as W
from ifgf_b200.autograd import matvec

KINDS = {
    "laplace": lambda c, k: G.LaplaceIfgfOperator(c["leaf"], c["order"]),
    "helmholtz": lambda c, k: G.HelmholtzIfgfOperator(k.real, c["leaf"], c["order"]),
    "modified": lambda c, k: G.ModifiedHelmholtzIfgfOperator(k, c["leaf"], c["order"]),
    "gradient": lambda c, k: G.GradHelmholtzIfgfOperator(k, c["leaf"], c["order"]),
    "double_layer": lambda c, k: G.DoubleLayerHelmholtzIfgfOperator(k, c["leaf"], c["order"]),
    "combined": lambda c, k: G.CombinedFieldHelmholtzIfgfOperator(k.real, c["leaf"], c["order"]),
}
GRAD_DX = 0            # derivative direction of the gradient kernel
TARGET_RADIUS = 1.25   # sphere of the targets when they are not the sources


def _case(name, kind, call, n, k_re, k_im, order, precision, *, m=0, surface="sphere", leaf=100,
          rhs=1):
    c = {"kind": kind, "call": call, "n": n, "m": m, "surface": surface, "k_re": k_re,
         "k_im": k_im, "leaf": leaf, "order": order, "precision": precision, "rhs": rhs}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a few thousand points, numpy in and out, as in a
        # script or in the iterations of a small boundary-element problem
        _case("helmholtz_4k_host", "helmholtz", "host", 4000, 16.0, 0.0, 8, "fp64", leaf=50),
        # plain Laplace, real densities, low order, one solver iteration
        _case("laplace_20k", "laplace", "device", 20000, 0.0, 0.0, 8, "fp64"),
        # high accuracy: an order above the common ones
        _case("helmholtz_30k_order12", "helmholtz", "device", 30011, 20.0, 0.0, 12, "fp64"),
        # the field of a solved density away from the surface: other targets
        # than sources, source normals, complex wavenumber
        _case("double_layer_field_60k", "double_layer", "device", 60013, 0.5, -20.0, 10, "fp64",
              m=20011),
        # medium frequency, FP64: the plain form at a size users start from
        _case("helmholtz_200k", "helmholtz", "device", 200000, 16 * math.pi, 0.0, 8, "fp64"),
        # the plain form at the headline size
        _case("helmholtz_1m", "helmholtz", "device", 1000000, 100.0, 0.0, 9, "fp64",
              surface="ellipsoid"),
        # one mixed matvec of an iterative solver, gradient kernel, odd size
        _case("gradient_50k_mixed", "gradient", "device", 50001, 0.25, -20.0, 9, "mixed"),
        # one mixed matvec at the headline size
        _case("helmholtz_1m_mixed", "helmholtz", "device", 1000000, 100.0, 0.0, 9, "mixed",
              surface="ellipsoid"),
        # eight right-hand sides at once, the headline's form at a size that
        # leaves room on the card (0.69 GB per 10,000 points with four planes)
        _case("helmholtz_600k_mixed_rhs8", "helmholtz", "batch", 600011, 78.0, 0.0, 9, "mixed",
              surface="ellipsoid", rhs=8),
        # many right-hand sides from host memory and back
        _case("helmholtz_100k_mixed_rhs16_host", "helmholtz", "batch_host", 100000, 20.0, 0.0, 9,
              "mixed", rhs=16),
        # a convolution-quadrature frequency set in one call
        _case("cq_100k_mixed_64k", "modified", "wavenumbers", 100000, 100.0, 0.0, 8, "mixed",
              rhs=64),
        # differentiation: a combined-field loss, its gradients by density and wavenumber
        _case("combined_100k_gradients", "combined", "gradients", 100000, 50.0, 0.0, 9, "fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above."""
    call = rng.choice(["host", "device", "device", "device", "batch", "batch_host", "wavenumbers",
                       "gradients"])
    leaf = rng.choice([50, 64, 100, 100, 128])
    surface = rng.choice(["sphere", "ellipsoid"])
    precision = rng.choice(["fp64", "mixed"])
    m, rhs = 0, 1
    if call == "wavenumbers":
        n, rhs = _log_int(rng, 5000, 100000), rng.randint(8, 64)
        return _case(None, "modified", call, n, 100.0, 0.0, rng.choice([8, 9]), "mixed",
                     leaf=leaf, rhs=rhs)
    if call == "gradients":
        n = _log_int(rng, 3000, 100000)
        kind = rng.choice(["combined", "helmholtz"])
        return _case(None, kind, call, n, rng.uniform(0.05, 0.16) * math.sqrt(n), 0.0,
                     rng.choice([8, 9]), "fp64", leaf=leaf)
    if call in ("batch", "batch_host"):
        n, rhs = _log_int(rng, 5000, 400000), rng.randint(2, 16)
        kind, precision, order = rng.choice(["helmholtz", "modified", "combined"]), "mixed", 9
        if n * rhs > 2000000:
            order = 8
    else:
        kind = rng.choice(sorted(KINDS))
        order = rng.choice([8, 9, 9, 10, 12])
        n = _log_int(rng, 2000, 40000 if order == 12 else 100000 if order == 10 else 400000)
        if rng.random() < 0.3:
            m = _log_int(rng, 1000, 50000)
    k = rng.uniform(0.04, 0.11) * math.sqrt(n)
    k_re, k_im = {"laplace": (0.0, 0.0), "helmholtz": (k, 0.0),
                  "combined": (k, 0.0)}.get(kind, (rng.uniform(0.1, 1.0), -k))
    return _case(None, kind, call, n, k_re, k_im, order, precision, m=m, surface=surface,
                 leaf=leaf, rhs=rhs)


def _points(case, seed):
    """Sources, targets and source normals (None if the kernel has none)."""
    axes = (1.0, 1.0, 1.0) if case["surface"] == "sphere" else (1.0, 1.0, 0.5)
    src = W.ellipsoid_points(case["n"], axes, seed)
    tgt = TARGET_RADIUS * W.sphere_points(case["m"], seed + 1) if case["m"] else src
    nrm = None
    if case["kind"] in ("double_layer", "combined"):
        nrm = src / np.asarray(axes)[:, None] ** 2
        nrm /= np.linalg.norm(nrm, axis=0)
    return src, tgt, nrm


def _wavenumbers(case):
    """BDF2 contour of convolution quadrature with step 0.01 (k_re = 1 / step)."""
    z = 0.9 * np.exp(2j * np.pi * np.arange(case["rhs"]) / case["rhs"])
    return (1.0 - 0.5 * z) * case["k_re"]


def _normal(seed, shape, real, mixed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(shape if real else tuple(shape) + (2,), generator=g, device="cuda",
                    dtype=torch.float32 if mixed else torch.float64).double()
    return w if real else torch.view_as_complex(w)


def _pinned(t):
    return t.cpu().pin_memory().numpy()


def prepare(case, seed):
    src, tgt, nrm = _points(case, seed)
    n, m = src.shape[1], tgt.shape[1]
    k = complex(case["k_re"], case["k_im"])
    op = KINDS[case["kind"]](case, k)
    if case["kind"] == "gradient":
        op.setDx(GRAD_DX)
    op.init(src, tgt, *(() if nrm is None else (nrm,)))
    mixed, real = case["precision"] == "mixed", case["kind"] == "laplace"
    if mixed:
        op.set_precision("mixed")
    s = {"call": case["call"], "op": op, "rhs": case["rhs"], "mixed": mixed, "real": real}
    batched = case["call"] in ("batch", "batch_host", "wavenumbers")
    w = _normal(seed, (case["rhs"], n) if batched else (n,), real, mixed)
    if case["call"] == "host":
        s["w"] = w.cpu().numpy()
    elif case["call"] == "batch_host":
        s["w"] = _pinned(w)
        s["u"] = _pinned(torch.zeros((case["rhs"], m), dtype=w.dtype))
    elif case["call"] == "gradients":
        s["w"], s["b"] = w, _normal(seed + 1, (m,), real, mixed)
        s["k"] = torch.tensor(case["k_re"], dtype=torch.float64, device="cuda",
                              requires_grad=True)
    else:
        s["w"] = w
        s["u"] = torch.empty((case["rhs"], m) if batched else (m,), dtype=w.dtype, device="cuda")
        if case["call"] == "wavenumbers":
            s["ks"] = _wavenumbers(case)
    return s


def run(s):
    op, call = s["op"], s["call"]
    if call == "host":
        u = op.mult(s["w"])
        return u.astype(np.float32 if s["real"] else np.complex64) if s["mixed"] else u
    if call == "batch_host":
        return op.mult_batch(s["w"], out=s["u"]).astype(np.float32 if s["real"] else np.complex64)
    if call == "gradients":
        x = s["w"].detach().requires_grad_()
        s["k"].grad = None
        u = matvec(op, x, s["k"])
        loss = 0.5 * (u - s["b"]).abs().square().sum()
        loss.backward()
        return {"u": u.detach(), "loss": loss.detach(), "dx": x.grad, "dk": s["k"].grad}
    w, u = s["w"].data_ptr(), s["u"].data_ptr()
    stream = torch.cuda.current_stream().cuda_stream
    if call == "device":
        op.mult_device(w, u, stream)
    elif call == "batch":
        op.mult_batch_device(w, u, s["rhs"], stream)
    else:
        op.mult_wavenumbers_device(s["ks"], w, u, stream)
    if s["mixed"]:
        return s["u"].to(torch.float32 if s["real"] else torch.complex64)
    return s["u"]


def work(case):
    """Points, densities and results once; the sums from the method's own counts.

    On a surface of n points a target meets about nine leaves of half-filled
    size directly and, on each of the log_4(n / leaf) levels above, a few
    dozen interpolants (of lo0 lo1 lo2 complex coefficients, 6 flops each) on
    the way up and at the targets."""
    n, m = case["n"], case["m"] or case["n"]
    p = case["order"]
    lo = (p - 6) * (p - 3) ** 2
    val = 8 if case["kind"] == "laplace" else 16
    passes = case["rhs"]
    if case["call"] == "gradients":  # u, A^H and dA/dk
        passes = 3
    levels = max(1.0, math.log(max(n, m) / case["leaf"], 4))
    flops = passes * (m * 9 * 0.5 * case["leaf"] * 23 + (n + m) * levels * 24 * 6 * lo)
    return {"bytes": 24.0 * (n + m) + passes * val * (n + m), "flops": flops}


# Pairs x planes of a dense sum that a B200 does in under 20 seconds.
EXACT_PAIRS = 4e11
TILE = 1 << 26


def _dense(case, k, src, tgt, nrm, w, what="A"):
    """Direct sums over all pairs in FP64: A w, A^H w or (dA/dk) w, by tiles of targets
    (w of shape (points,) or (points, right-hand sides))."""
    dev = "cuda"
    x = torch.from_numpy(src).to(dev)
    y = torch.from_numpy(tgt).to(dev)
    nv = None if nrm is None else torch.from_numpy(nrm).to(dev)
    n, m = x.shape[1], y.shape[1]
    kind = case["kind"]
    real = kind == "laplace"
    out = torch.zeros((n if what == "AH" else m,) + w.shape[1:], dtype=w.dtype, device=dev)
    step = max(1, TILE // n)
    for t0 in range(0, m, step):
        t1 = min(m, t0 + step)
        d = [x[j][None, :] - y[j, t0:t1, None] for j in range(3)]
        r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt_()
        inv = torch.where(r < 1e-12, torch.zeros_like(r), 1.0 / r)
        if real:
            out[t0:t1] = (inv @ w) / (4 * math.pi)
            continue
        if kind in ("helmholtz", "combined"):
            e = torch.polar(inv, k.real * r)
        else:
            e = torch.polar(inv * torch.exp(-k.real * r), -k.imag * r)
        if kind == "gradient":
            e *= torch.complex((k.real + inv) * inv, k.imag * inv) * d[GRAD_DX]
        elif kind == "double_layer":
            xn = d[0] * nv[0] + d[1] * nv[1] + d[2] * nv[2]
            e *= torch.complex((k.real + inv) * inv, k.imag * inv) * xn
        elif kind == "combined":
            nxy = -(d[0] * nv[0] + d[1] * nv[1] + d[2] * nv[2])
            if what == "dA/dk":
                e *= torch.complex(k.real * (nxy + r), torch.full_like(r, -1.0))
            else:
                e *= torch.complex(nxy * inv * inv, -k.real * (nxy * inv + 1.0) * (inv > 0))
        elif what == "dA/dk":
            e *= 1j * r
        if what == "AH":
            out += e.conj().T @ w[t0:t1]
        else:
            out[t0:t1] = e @ w
    return out if real else out / (4 * math.pi)


def exact(case, seed):
    n, m = case["n"], case["m"] or case["n"]
    passes = {"gradients": 3, "wavenumbers": case["rhs"]}.get(case["call"], 1)
    if float(n) * m * passes > EXACT_PAIRS:
        return None
    src, tgt, nrm = _points(case, seed)
    k = complex(case["k_re"], case["k_im"])
    mixed, real = case["precision"] == "mixed", case["kind"] == "laplace"
    if case["call"] == "wavenumbers":
        w = _normal(seed, (case["rhs"], n), real, mixed)
        return torch.stack([_dense(case, complex(kp), src, tgt, nrm, w[p])
                            for p, kp in enumerate(_wavenumbers(case))])
    if case["call"] in ("batch", "batch_host"):
        w = _normal(seed, (case["rhs"], n), real, mixed)
        return _dense(case, k, src, tgt, nrm, w.T.contiguous()).T.contiguous()
    w = _normal(seed, (n,), real, mixed)
    u = _dense(case, k, src, tgt, nrm, w)
    if case["call"] != "gradients":
        return u
    g = u - _normal(seed + 1, (m,), real, mixed)
    dk = torch.vdot(g, _dense(case, k, src, tgt, nrm, w, "dA/dk")).real
    return {"u": u, "loss": 0.5 * g.abs().square().sum(),
            "dx": _dense(case, k, src, tgt, nrm, g, "AH"), "dk": dk}
