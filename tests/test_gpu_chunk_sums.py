"""FP64 sums of like-signed terms over many chunks of sources, against extended
precision: few targets, so that the sources are cut into chunks of 64.

Tolerance, root mean square over the targets and relative: 80 chunk sums join the
running sum eight at a time, ten roundings of at most 2^-53 (0.58 of it rms) on partial
sums that grow to the whole one (their rms 0.58 of it), 1.2e-16; a chunk's own sum, an
eightieth of the whole, adds less than 1e-17, the constants three roundings, 1.1e-16:
2e-16, and half of that again for the sample: 3e-16."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["FP64", "FP64_CHORD"])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_like_signed_plane_sums(gpu_ctx, prec, eps):
    rng = np.random.default_rng(5)
    ns, nt = 5000, 150
    y, x, g = rng.uniform(-2, 2, (ns, 2)), rng.uniform(-2, 2, (nt, 2)), rng.uniform(0.5, 1, ns)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    u = torch.empty(nt, 2, dtype=torch.float64, device="cuda")
    p = torch.empty(nt, dtype=torch.float64, device="cuda")
    gpu_ctx.set_precision(getattr(core, prec))
    F.ic2d_passive_sums(gpu_ctx, u, p, dev(x), dev(y), dev(g), dev(np.ones(ns)),
                        dev(np.zeros(ns, np.uint8)), eps)
    gpu_ctx.synchronize()
    gpu_ctx.set_precision(core.FP64)
    ld = np.longdouble
    pi = ld("3.14159265358979323846264338327950288")
    ur, pr = np.zeros((nt, 2), ld), np.zeros(nt, ld)
    for i, t in enumerate(x.astype(ld)):
        d = t - y.astype(ld)
        q = (d * d).sum(1) + ld(eps * eps)
        w = ((g / q)[:, None] * d).sum(0) / (2 * pi)
        ur[i] = -w[1], w[0]
        pr[i] = -(g * np.log(q)).sum() / (4 * pi)
    rms = lambda a: np.sqrt((np.asarray(a, np.float64) ** 2).mean())
    assert rms(u.cpu().numpy() - ur) <= 3e-16 * rms(ur)
    assert rms(p.cpu().numpy() - pr) <= 3e-16 * rms(pr)
