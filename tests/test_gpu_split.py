"""The LPM_FP64 sphere sums on the FP32 pipe (nbody_split) at the sizes and
inputs where they can go wrong, against the FP64 oracle: tile and target-block
remainders, the least source count, the target's own source, stage positions
off the sphere, near and coincident pairs, targets far outside the sources'
range, strengths of any scale, eps from none to larger than the domain.

Tolerance 1e-12 of the largest reference value, the FP64 parity tolerance of
the other tests.  The oracle's 1 - x.y is off by 1e-16 / (1 - x.y) of a pair,
so where eps = 0 lets pairs come arbitrarily close the reference is the same sum
with 1 - x.y = |x - y|^2 / 2 + (1 - |x|^2) / 2 + (1 - |y|^2) / 2."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _points(rng, n, drift=0.0):
    x = rng.normal(size=(n, 3))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    return x * (1 + drift * rng.uniform(-1, 1, (n, 1)))


def _spread(n, drift, rng):
    """n points of a Fibonacci spiral (no two close), radii off by drift."""
    i = np.arange(n) + 0.5
    z = 1 - 2 * i / n
    p = np.pi * (1 + 5**0.5) * i
    r = np.sqrt(1 - z * z)
    x = np.stack([r * np.cos(p), r * np.sin(p), z], 1)
    return x * (1 + drift * rng.uniform(0, 1, (n, 1)))


def _rel(got, ref):
    got, ref = got.cpu().numpy(), np.asarray(ref)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    f = np.isfinite(ref)
    return np.abs(got[f] - ref[f]).max() / np.abs(ref[f]).max()


def _reference(oracle, x, y, z, a, m, eps, self_rule=0):
    """(u, psi): the oracle for eps > 0, the well-conditioned sum for eps = 0."""
    if eps > 0 and self_rule:
        return oracle.ic2d_active_sums(y, z, a, m, eps, self_rule=1)
    if eps > 0:
        return oracle.ic2d_passive_sums(x, y, z, a, m, eps)
    half = lambda p: ((1 - (p.astype(np.longdouble) ** 2).sum(1)) / 2).astype(np.float64)
    keep = m == 0
    ys, g, hy = y[keep], (z * a)[keep], half(y)[keep]
    slot = np.flatnonzero(keep)
    u, p = np.zeros((len(x), 3)), np.zeros(len(x))
    for i, (xi, hx) in enumerate(zip(x, half(x))):
        d = xi - ys
        q = 0.5 * (d * d).sum(1) + (hx + hy)
        ok = slot != i if self_rule else slice(None)
        w = ((g / np.where(q == 0, 1, q))[:, None] * d)[ok].sum(0)
        u[i] = np.cross(xi, w) / (4 * np.pi)
        p[i] = -(g[ok] * np.log(np.where(q == 0, 1, q)[ok])).sum() / (4 * np.pi)
    return u, p


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _run(ctx, x, y, z, a, m, eps, collocated=False):
    ctx.set_precision(core.FP64)
    X, Y, Z, A, M = (_dev(v) for v in (x, y, z, a, m))
    u = torch.zeros(len(x), 3, dtype=torch.float64, device="cuda")
    p = torch.zeros(len(x), dtype=torch.float64, device="cuda")
    if collocated:
        F.ic2d_active_sums(ctx, u, p, Y, Z, A, M, eps, self_rule=1)
    else:
        F.ic2d_passive_sums(ctx, u, p, X, Y, Z, A, M, eps)
    ctx.synchronize()
    return u, p


@pytest.mark.parametrize("nsrc,ntgt", [(1024, 1024), (1025, 977), (1151, 1000), (1153, 1025),
                                       (4097, 257), (2047, 4099)])
@pytest.mark.parametrize("eps", [0.0, 0.03])
def test_sizes(gpu_ctx, oracle, nsrc, ntgt, eps):
    rng = np.random.default_rng(nsrc)
    y, x = _spread(nsrc, 0.0, rng), _spread(ntgt, 0.0, rng)[:, [1, 2, 0]]
    z, a, m = rng.normal(size=nsrc), np.full(nsrc, 4 * np.pi / nsrc), np.zeros(nsrc, np.uint8)
    m[rng.permutation(nsrc)[: max(0, nsrc - 1024) // 3]] = 1
    u, p = _run(gpu_ctx, x, y, z, a, m, eps)
    ur, pr = _reference(oracle, x, y, z, a, m, eps)
    assert _rel(u, ur) < TOL and _rel(p, pr) < TOL


@pytest.mark.parametrize("eps", [0.0, 0.02])
@pytest.mark.parametrize("drift", [0.0, 1e-4])
def test_own_source_and_drift(gpu_ctx, oracle, eps, drift):
    """Collocated targets skip their own source, on and off the sphere."""
    rng = np.random.default_rng(3)
    n = 1500
    y = _spread(n, drift, rng)
    z, a, m = rng.normal(size=n), np.full(n, 4 * np.pi / n), np.zeros(n, np.uint8)
    m[::17] = 1
    u, p = _run(gpu_ctx, y, y, z, a, m, eps, collocated=True)
    ur, pr = _reference(oracle, y, y, z, a, m, eps, self_rule=1)
    # a masked slot's own point is no source; every target is compared
    assert _rel(u, ur) < TOL and _rel(p, pr) < TOL


@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e+190])
def test_near_and_coincident(gpu_ctx, oracle, scale):
    """Targets 0.02 from a source and exactly on one (eps keeps it finite),
    strengths of any scale (outside 2^+-400: the FP64 path)."""
    rng = np.random.default_rng(5)
    n = 2000
    y = _spread(n, 0.0, rng)
    t = np.cross(y, [0.3, -0.5, 0.8])
    near = y[:400] + 0.02 * t[:400] / np.linalg.norm(t[:400], axis=1, keepdims=True)
    near /= np.linalg.norm(near, axis=1, keepdims=True)
    x = np.concatenate([near, y[500:700], _spread(300, 0.0, rng)])
    z, a, m = rng.normal(size=n) * scale, np.full(n, 4 * np.pi / n), np.zeros(n, np.uint8)
    for eps in (0.01, 0.3):
        u, p = _run(gpu_ctx, x, y, z, a, m, eps)
        ur, pr = oracle.ic2d_passive_sums(x, y, z, a, m, eps)
        assert _rel(u, ur) < TOL and _rel(p, pr) < TOL


@pytest.mark.parametrize("rx,ry,eps", [(0.5, 1.0, 0.01), (0.98, 1.0, 0.1), (1.0, 0.9, 0.01),
                                       (40.0, 1.0, 7.0), (3.0, 1.0, 2.0)])
def test_off_the_sphere(gpu_ctx, oracle, rx, ry, eps):
    """Targets or sources off the sphere (pairs, targets or all on FP64; targets of
    40 also out of the scaled range), mixed with targets on it; 1 - x.y + eps^2
    stays above 0.02, so the tolerance holds."""
    rng = np.random.default_rng(8)
    y, x = ry * _spread(1300, 0.0, rng), _spread(1200, 0.0, rng)[:, [1, 2, 0]]
    x[200:700] *= rx
    z, a, m = rng.normal(size=1300), np.full(1300, 0.01), np.zeros(1300, np.uint8)
    sel = slice(None) if eps > 0.05 or ry < 1 else slice(200, 700)  # no close pairs
    u, p = _run(gpu_ctx, x, y, z, a, m, eps)
    ur, pr = oracle.ic2d_passive_sums(x, y, z, a, m, eps)
    assert _rel(u[sel], ur[sel]) < TOL and _rel(p[sel], pr[sel]) < TOL


@pytest.mark.parametrize("eps", [3.0, 1e4])
def test_large_eps(gpu_ctx, oracle, eps):
    """eps beyond the domain: still split, then (1e4) FP64 throughout."""
    rng = np.random.default_rng(6)
    y, x = _spread(1100, 0.0, rng), _spread(1000, 0.0, rng)[:, [2, 0, 1]]
    z, a, m = rng.normal(size=1100), np.full(1100, 0.01), np.zeros(1100, np.uint8)
    u, p = _run(gpu_ctx, x, y, z, a, m, eps)
    ur, pr = oracle.ic2d_passive_sums(x, y, z, a, m, eps)
    assert _rel(u, ur) < TOL and _rel(p, pr) < TOL


@pytest.mark.parametrize("nsrc,ntgt", [(1, 1), (7, 65), (8, 64), (9, 63), (1023, 130), (320, 162)])
def test_small_grids(gpu_ctx, oracle, nsrc, ntgt):
    """The one-target-per-thread FP64 grid at its tile and block remainders,
    sphere and plane."""
    rng = np.random.default_rng(nsrc + ntgt)
    y, x = _spread(nsrc, 0.0, rng), _spread(ntgt, 0.0, rng)[:, [1, 2, 0]]
    z, a, m = rng.normal(size=nsrc), np.full(nsrc, 4 * np.pi / nsrc), np.zeros(nsrc, np.uint8)
    u, p = _run(gpu_ctx, x, y, z, a, m, 0.05)
    ur, pr = oracle.ic2d_passive_sums(x, y, z, a, m, 0.05)
    assert _rel(u, ur) < TOL and _rel(p, pr) < TOL
    x2, y2 = x[:, :2].copy(), y[:, :2].copy()
    u2 = torch.zeros(ntgt, 2, dtype=torch.float64, device="cuda")
    p2 = torch.zeros(ntgt, dtype=torch.float64, device="cuda")
    F.ic2d_passive_sums(gpu_ctx, u2, p2, _dev(x2), _dev(y2), _dev(z), _dev(a), _dev(m), 0.05)
    gpu_ctx.synchronize()
    ur, pr = oracle.ic2d_passive_sums(x2, y2, z, a, m, 0.05)
    assert _rel(u2, ur) < TOL and _rel(p2, pr) < TOL
