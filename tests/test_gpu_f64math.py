"""Reciprocal, logarithm and exponential of the FP64 pair loops, through the sums:
one source at the origin and targets at chosen distances, so that an output is
the function's value times constants.  Arguments at the seams of the tables, at
powers of two, beside 1, and from the largest to the smallest that the fixed-point
forms take and beyond.

Tolerances, in units of 2^-53 of the value: reciprocal at most 2 and two products,
6; logarithm at most 8 (five roundings of parts up to twice the value, and
2^-67 / 2^-16 next to 1) and three factors, 12 (14 with the base-2 factor of the
chord form); exponential 2, its argument exact to 2^-54, the cubic's
Horner steps 6 and three factors: 12 of the cubic's absolute terms."""
import math
from fractions import Fraction

import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu

ULP = 2.0**-53


def _args():
    """|d|^2 wanted: seams, powers of two, values beside 1, a wide range."""
    k = np.arange(0, 4097, 64)
    seams = np.concatenate([1 + k / 4096, 1 + (k + 0.5) / 4096])
    near = 2.0 ** -np.arange(4, 53)
    wide = 10.0 ** np.arange(-290, 291, 10.0)
    root = math.sqrt(2) * (1 + np.arange(-4, 5) * 2.0**-52)
    one = np.concatenate([1 + near, 1 - near])
    return np.concatenate([seams, 0.25 * seams, 7.0 * seams, one, wide, root, 2.0 ** np.arange(-40, 41)])


def _targets(args, c0=0.0):
    """d and the rounded d^2 + c0 that the kernel's argument is."""
    d = np.sqrt(args)
    return d, np.array([float(Fraction(v) ** 2 + Fraction(c0)) for v in d])


@pytest.mark.parametrize("prec", ["FP64", "FP64_CHORD"])
@pytest.mark.parametrize("n", [1, 63, 0])
def test_reciprocal_and_logarithm(gpu_ctx, prec, n):
    a = _args()
    if prec == "FP64_CHORD":
        a = a[a > 1e-10]  # its 1e-30 beside |d|^2
    d, q = _targets(a[:n] if n else a, 1e-30 if prec == "FP64_CHORD" else 0.0)
    x = torch.from_numpy(np.stack([d, 0 * d], 1)).cuda()
    y = torch.zeros(1, 2, dtype=torch.float64, device="cuda")
    one, m = torch.ones(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.uint8, device="cuda")
    u, psi = torch.empty_like(x), torch.empty(len(d), dtype=torch.float64, device="cuda")
    gpu_ctx.set_precision(getattr(core, prec))
    F.ic2d_passive_sums(gpu_ctx, u, psi, x, y, one, one, m, 0.0)
    gpu_ctx.synchronize()
    gpu_ctx.set_precision(core.FP64)
    ru = np.asarray(1 / (2 * np.longdouble(math.pi) * q) * d, dtype=np.float64)
    rp = np.asarray(-np.log(q.astype(np.longdouble)) / (4 * np.longdouble(math.pi)), dtype=np.float64)
    assert (np.abs(u[:, 1].cpu().numpy() - ru) <= 6 * ULP * np.abs(ru)).all()
    assert (np.abs(psi.cpu().numpy() - rp) <= (14 if prec == "FP64_CHORD" else 12) * ULP * np.abs(rp)).all()


@pytest.mark.parametrize("n", [1, 129, 3000])
def test_exponential(gpu_ctx, n):
    d, _ = _targets(np.concatenate([np.linspace(0, 745.9, n), [0.0, 1e-30, 1e-9, math.log(2), 708.0, 745.5, 800.0]]))
    nt = len(d)
    x = torch.from_numpy(np.stack([d, 0 * d], 1)).cuda()
    y = torch.full((1, 2), 0.0, dtype=torch.float64, device="cuda")
    one, z = torch.ones(1, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    m = torch.zeros(1, dtype=torch.uint8, device="cuda")
    gpu_ctx.set_precision(core.FP64)
    o = F.swe_plane_vertex_sums(gpu_ctx, x, torch.zeros(nt, dtype=torch.float64, device="cuda"), y, z, z, one, m,
                                one, 0.5, 1.0)
    gpu_ctx.synchronize()
    L = d.astype(np.longdouble) ** 2  # the kernel's |d|^2 keeps 62 bits
    e = np.exp(-L) / np.longdouble(math.pi)
    ref = (40 - 40 * L + 10 * L * L - 2 * L**3 / 3) * e
    tol = 12 * ULP * (40 + 40 * L + 10 * L * L + 2 * L**3 / 3) * e + 1e-320
    assert (np.abs(o["laps"].cpu().numpy() - ref) <= tol).all()
