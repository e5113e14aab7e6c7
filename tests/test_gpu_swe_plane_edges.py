"""The FP64 planar SWE sums at values that are not finite and at pairs nearly along
an axis, where one component of d is far smaller than the other.

Tolerance of the components, in units of 2^-53 of each: |d|^2 + eps^2 and its
reciprocal 3, the products and the constants 3 for a velocity; twice that and two
sums for a gradient: 6 and 14."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu

ULP = 2.0**-53
COLS = {"du1dx1": 2, "du1dx2": 3, "du2dx1": 4, "du2dx2": 5, "laps": 6, "psi": 7, "phi": 8}


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _sums(ctx, x, sx, y, z, g, a, sy, eps, pse):
    ctx.set_precision(core.FP64)
    o = F.swe_plane_vertex_sums(ctx, _dev(x), _dev(sx), _dev(y), _dev(z), _dev(g), _dev(a),
                                _dev(np.zeros(len(y), np.uint8)), _dev(sy), eps, pse)
    ctx.synchronize()
    return {k: v.cpu().numpy() for k, v in o.items()}


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["source height", "target height", "area", "position"])
def test_not_finite(gpu_ctx, oracle, value, where):
    """Where the outputs are NaN or infinite, as the reference's: the smoothing kernel
    of most pairs here is 0, and 0 times such a value is NaN."""
    rng = np.random.default_rng(4)
    x, y = rng.uniform(-3, 3, (150, 2)), rng.uniform(-3, 3, (90, 2))
    sx, sy = rng.normal(size=150), rng.normal(size=90)
    z, g, a = rng.normal(size=90), rng.normal(size=90), rng.uniform(0.5, 1, 90)
    if where == "source height":
        sy[40] = value
    elif where == "target height":
        sx[70] = value
    elif where == "area":
        a[40] = value
    else:
        y[40, 0] = value
    o = _sums(gpu_ctx, x, sx, y, z, g, a, sy, 0.02, 0.05)
    r = oracle.swe_plane_sums(x, sx, y, z, g, a, np.zeros(90, np.uint8), sy, 0.02, 0.05)
    for k, c in COLS.items():
        assert np.array_equal(np.isfinite(o[k]), np.isfinite(r[:, c])), k
        if where != "area":  # infinite strengths: infinity or NaN as the terms are added
            assert np.array_equal(np.isnan(o[k]), np.isnan(r[:, c])), k


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("eps", [0.0, 0.01])
def test_nearly_along_an_axis(gpu_ctx, swap, eps):
    ld = np.longdouble
    k = np.arange(0, 300)
    x = np.stack([0.7 * (1 + 0.001 * k), -1.3 * 2.0 ** -(k / 3.0)], 1)
    x = np.concatenate([x, [[0.7, 1e-250], [0.7, 5e-324], [0.7, 0.0]]])
    if swap:
        x = x[:, ::-1].copy()
    y, one, zero = np.zeros((1, 2)), np.ones(1), np.zeros(1)
    o = _sums(gpu_ctx, x, np.zeros(len(x)), y, one, zero, one, zero, eps, 1.0)
    d0, d1 = x.astype(ld).T
    R = d0 * d0 + d1 * d1 + ld(eps) * ld(eps)
    pi = ld("3.14159265358979323846264338327950288")

    def near(got, ref, tol):
        return (np.abs(got - ref) <= tol * ULP * np.abs(ref) + 1e-300).all()

    assert near(o["u"][:, 0], -d1 / (2 * pi * R), 6) and near(o["u"][:, 1], d0 / (2 * pi * R), 6)
    assert near(o["du1dx1"], d0 * d1 / (pi * R * R), 14)
    assert near(o["du2dx2"], -d0 * d1 / (pi * R * R), 14)
