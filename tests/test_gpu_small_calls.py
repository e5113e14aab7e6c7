"""Functor calls of few slots, whose sources are compacted and packed by one launch
without a host read of their count: sizes around its thread blocks and its limit
(32,768 slots), masks that leave a prefix, alternate slots, one source or none, and a
target at the origin, where padding records lie.

Tolerance against plain FP64 sums, of the largest value: 1e-12 for the FP64 forms; FP32C
2e-6 for velocity and stream function, as the other FP32C tests."""
import math

import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu


def _masks(n):
    k = np.arange(n)
    return {"none": k < 0, "prefix": k < n // 2, "alternate": k % 2 == 1, "but one": k != n - 1, "all": k >= 0}


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1025, 32768, 32769])
@pytest.mark.parametrize("prec", ["FP64", "FP64_CHORD", "FP64_EXACT", "FP32C"])
def test_small_calls(gpu_ctx, n, prec):
    rng = np.random.default_rng(n)
    y, g, a = rng.uniform(-2, 2, (n, 2)), rng.normal(size=n), rng.uniform(0.5, 1.0, n) / n
    x = np.concatenate([[[0.0, 0.0]], rng.uniform(-2, 2, (32, 2))])
    eps = 0.1
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()  # noqa: E731
    d = x[:, None] - y[None]
    R = (d**2).sum(2) + eps * eps
    gpu_ctx.set_precision(getattr(core, prec))
    tol = 2e-6 if prec == "FP32C" else 1e-12
    for name, mask in _masks(n).items():
        w = np.where(mask, 0.0, g * a)
        u, psi = torch.full((33, 2), 7.0, dtype=torch.float64).cuda(), torch.full((33,), 7.0, dtype=torch.float64).cuda()
        F.ic2d_passive_sums(gpu_ctx, u, psi, dev(x), dev(y), dev(g), dev(a), dev(mask.astype(np.uint8)), eps)
        gpu_ctx.synchronize()
        q = w / R
        ru = np.stack([-(q * d[..., 1]).sum(1), (q * d[..., 0]).sum(1)], 1) / (2 * math.pi)
        rp = -(w * np.log(R)).sum(1) / (4 * math.pi)
        # cancelling sums: errors scale with the sums of sizes
        su = np.abs(q[..., None] * d).sum(1).max() / (2 * math.pi)
        sp = np.abs(w * np.log(R)).sum(1).max() / (4 * math.pi)
        assert np.abs(u.cpu().numpy() - ru).max() <= tol * su, name
        assert np.abs(psi.cpu().numpy() - rp).max() <= tol * sp, name
    gpu_ctx.set_precision(core.FP64)
