"""The FP64 spherical SWE sums against the same sums in extended precision: eps from
a mesh spacing to far beyond the sphere, strengths of both signs and of one, targets
on and off the sphere and at its centre.

Tolerances, of an output's largest value.  A term is good to about 10 roundings, and
the running sums' roundings add up as sqrt(200) of 2^-53 on partial sums up to a few
times the result: 1e-14 (velocity and gradient), twice that and the squares' own
cancellation for the double dot product, 4e-14.  1 - x.y + eps^2 stays above 0.1,
which keeps its own rounding, 1e-16, below that."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _cross(a, b):
    return np.stack([a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1],
                     a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2],
                     a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]], -1)


def _reference(x, y, rot, pot, eps):
    """u, M and M : M^T, term by term: u = c rot + w pot over 4 pi D,
    M = (D [y]x + c v^T) rot - (v w^T + D s P) pot over 4 pi D^2."""
    ld = np.longdouble
    x, y, rot, pot = (v.astype(ld) for v in (x, y, rot, pot))
    e2, pi4 = ld(eps * eps), 4 * ld("3.14159265358979323846264338327950288")
    X, Y = x[:, None, :], y[None, :, :]
    s = (X * Y).sum(-1)
    D = 1 - s + e2
    c, w, v = _cross(X, Y), Y - s[..., None] * X, (1 + e2) * X - Y
    sz, ss = rot / (pi4 * D), pot / (pi4 * D)
    u = (c * sz[..., None] + w * ss[..., None]).sum(1)
    M = np.einsum("ij,ija,ijb->iab", sz / D, c, v) - np.einsum("ij,ija,ijb->iab", ss / D, v, w)
    z = (sz[..., None] * Y).sum(1)
    K = np.zeros_like(M)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -z[:, 2], z[:, 1], -z[:, 0]
    K[:, 1, 0], K[:, 2, 0], K[:, 2, 1] = z[:, 2], -z[:, 1], z[:, 0]
    P = np.eye(3) - x[:, :, None] * x[:, None, :]
    M = M + K - (ss * s).sum(1)[:, None, None] * P
    return u, M, np.einsum("iab,iba->i", M, M)


@pytest.mark.parametrize("eps", [0.4, 1.0, 3.0, 10.0, 1e2, 1e4, 1e8])
@pytest.mark.parametrize("same_sign", [False, True])
@pytest.mark.parametrize("off", [False, True])
def test_gradient(gpu_ctx, eps, same_sign, off):
    rng = np.random.default_rng(11)
    unit = lambda p: p / np.linalg.norm(p, axis=1, keepdims=True)
    y = unit(rng.normal(size=(200, 3)))
    x = unit(rng.normal(size=(4000, 3)))
    if off:
        x[:2000] *= rng.uniform(0.05, 1.5, (2000, 1))
        x[7], x[8] = 0.0, 1e-9 * x[8]
    x = x[(1 - x @ y.T).min(1) + eps * eps > 0.1]
    assert 60 < len(x)
    z, g, a = rng.normal(size=200), rng.normal(size=200), np.full(200, 0.02)
    if same_sign:
        z, g = np.abs(z), np.abs(g)
    gpu_ctx.set_precision(core.FP64)
    o = F.swe_sphere_vertex_sums(gpu_ctx, _dev(x), _dev(y), _dev(z), _dev(g), _dev(a),
                                 _dev(np.zeros(200, np.uint8)), eps, want_grad=True)
    gpu_ctx.synchronize()
    u, M, dd = _reference(x, y, -z * a, -g * a, eps)
    near = lambda got, ref: np.abs(got.cpu().numpy().reshape(ref.shape) - ref).max() / np.abs(ref).max()
    assert near(o["u"], u) < 1e-14
    assert near(o["grad"], M) < 1e-14
    assert near(o["ddot"], dd) < 4e-14
