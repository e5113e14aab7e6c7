"""LPM_FP64 sphere sums over at least 1,024 sources whose strengths are not of like
size and sign: a few strong ones seen from afar, a compact cluster of random signs,
infinite and NaN strengths.

A pair 90 degrees and more apart has 1 - x.y in [1, 2], formed by three roundings of
at most 1.1e-16, its reciprocal and quotient two more: 5.5e-16 of the term.  The cross
product with x adds three, the running sum of 20 terms at most 20 on partial sums that
grow to the whole one, 1.1e-15: 2e-15 of the terms' sum of magnitudes in all."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu


def _spread(n):
    i = np.arange(n) + 0.5
    z = 1 - 2 * i / n
    p = np.pi * (1 + 5**0.5) * i
    r = np.sqrt(1 - z * z)
    return np.stack([r * np.cos(p), r * np.sin(p), z], 1)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _sums(ctx, x, y, g, eps=0.0):
    ctx.set_precision(core.FP64)
    one, m = np.ones(len(y)), np.zeros(len(y), np.uint8)
    u = torch.empty(len(x), 3, dtype=torch.float64, device="cuda")
    p = torch.empty(len(x), dtype=torch.float64, device="cuda")
    F.ic2d_passive_sums(ctx, u, p, _dev(x), _dev(y), _dev(g), _dev(one), _dev(m), eps)
    ctx.synchronize()
    return u.cpu().numpy(), p.cpu().numpy()


def _reference(x, y, g):
    """u, psi and the sums of magnitudes that their errors are measured by."""
    ld = np.longdouble
    x, y, g = (v.astype(ld) for v in (x, y, g))
    arg = 1 - x @ y.T
    k = 1 / (4 * ld("3.14159265358979323846264338327950288"))
    w = (g / arg) @ y
    u = -k * np.stack([x[:, 1] * w[:, 2] - x[:, 2] * w[:, 1], x[:, 2] * w[:, 0] - x[:, 0] * w[:, 2],
                       x[:, 0] * w[:, 1] - x[:, 1] * w[:, 0]], 1)
    return u, -k * (np.log(arg) @ g), k * (np.abs(g) / arg).sum(1), k * (np.abs(np.log(arg)) @ np.abs(g))


@pytest.mark.parametrize("strong", [1, 5, 20])
@pytest.mark.parametrize("signs", ["like", "random"])
@pytest.mark.parametrize("n", [1024, 4100])
def test_few_sources_of_strength(gpu_ctx, strong, signs, n):
    rng = np.random.default_rng(strong)
    y = _spread(n)  # the first are the nearest to the pole
    g = np.zeros(n)
    g[:strong] = rng.uniform(0.5, 1.0, strong) * (rng.choice([-1, 1], strong) if signs == "random" else 1)
    x = _spread(2000)[:, [1, 2, 0]]
    x = x[(x @ y[:strong].T).max(1) < 0]
    u, p = _sums(gpu_ctx, x, y, g)
    ur, pr, su, sp = _reference(x, y, g)
    assert (np.abs(u - ur).max(1) <= 2e-15 * su).all()
    assert (np.abs(p - pr) <= 2e-15 * (sp + su)).all()


@pytest.mark.parametrize("n", [4100, 20000])
def test_compact_cluster_of_random_signs(gpu_ctx, n):
    """A cap of 1 / 20 of the sources, as strong as each other, cancelling: the error
    against the sum of FP64 pair errors, 4e-16 of sqrt(sum t^2), twelve times."""
    rng = np.random.default_rng(3)
    y = _spread(n)
    k = n // 20
    g = np.zeros(n)
    g[:k] = rng.choice([-1.0, 1.0], k)
    x = _spread(1500)[:, [1, 2, 0]]
    x = x[(x @ y[:k].T).max(1) < 0]
    u, _ = _sums(gpu_ctx, x, y, g)
    ur = _reference(x, y, g)[0]
    t2 = ((g / (1 - x @ y.T)) ** 2).sum(1)
    assert (np.abs(u - ur).max(1) <= 12 * 4e-16 * np.sqrt(t2) / (4 * np.pi)).all()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("eps", [0.0, 0.1])
def test_strength_not_finite(gpu_ctx, value, eps):
    """As the same call with a few sources: infinite values stay infinite."""
    y = _spread(1500)
    g = np.full(1500, 0.01)
    g[700] = value
    x = _spread(1100)[:, [1, 2, 0]]
    u, p = _sums(gpu_ctx, x, y, g, eps)
    uf, pf = _sums(gpu_ctx, x, y[690:710], g[690:710], eps)
    assert np.array_equal(np.isnan(p), np.isnan(pf))
    assert np.array_equal(p[~np.isfinite(p)], pf[~np.isfinite(pf)], equal_nan=True)
    assert np.array_equal(np.isnan(u), np.isnan(uf))
    assert np.array_equal(u[np.isinf(u)], uf[np.isinf(uf)])
