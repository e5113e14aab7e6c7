"""The stream function of LPM_FP64 sphere sums over 1,280 and more sources with the
velocity beside it: a Rossby-Haurwitz wave, whose terms cancel, against extended
precision.

Tolerance, of the largest value: 1 - x.y is off by 3.3e-16 (three roundings below 2), the
logarithm by that over 1 - x.y, 3e-15 at the closest pairs and 7e-16 rms over the sphere;
n terms g log add up to 7e-16 sqrt(sum g^2) / (4 pi), 3e-17 and less of psi's scale here;
the running sums' roundings are at most 2^-53 of partial sums up to the tile's and the
chunks', a few times psi: 1e-15."""
import math

import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F
from lpm_gb300.bve import rossby_haurwitz_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,n", [(3, 1280), (4, 5120)])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_rossby_haurwitz_stream_function(gpu_ctx, level, n, eps):
    vx, fx, fa, fm = core.build_mesh(core.MESH_ICOS_TRI, level, 1.0)
    y, a = fx[fm == 0], fa[fm == 0]
    assert len(y) == n
    z = core.eval_ic(core.IC_RH54, rossby_haurwitz_params(), y)
    q, _ = np.linalg.qr(np.random.default_rng(level).normal(size=(3, 3)))
    y, x = y @ q, vx @ q
    y, x = (p / np.linalg.norm(p, axis=1, keepdims=True) for p in (y, x))
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    u = torch.empty(len(x), 3, dtype=torch.float64, device="cuda")
    p = torch.empty(len(x), dtype=torch.float64, device="cuda")
    gpu_ctx.set_precision(core.FP64)
    F.ic2d_passive_sums(gpu_ctx, u, p, dev(x), dev(y), dev(z), dev(a), dev(np.zeros(n, np.uint8)), eps)
    gpu_ctx.synchronize()
    p = p.cpu().numpy()
    ld = np.longdouble
    ys, g = y.astype(ld), (z * a).astype(ld)
    hy = 1 - (ys * ys).sum(1)
    idx = np.random.default_rng(1).choice(len(x), 200, False)
    ref = np.zeros(200, ld)
    for k, i in enumerate(idx):
        t = x[i].astype(ld)
        d = t - ys
        arg = ((d * d).sum(1) + hy + (1 - (t * t).sum())) / 2 + ld(eps * eps)
        ref[k] = -(g * np.log(arg)).sum() / (4 * ld(math.pi))
    assert np.abs(p[idx] - ref).max() <= 1e-15 * np.abs(ref).max()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_target_not_finite(gpu_ctx, value, eps):
    """A target that is not finite: its sums are those of a call of the same sources over
    that target and three others (few pairs: FP64 throughout), the others' are finite."""
    vx, fx, fa, fm = core.build_mesh(core.MESH_ICOS_TRI, 3, 1.0)
    y, a = fx[fm == 0], fa[fm == 0]
    x = vx[:600].copy()
    x[77, 1] = value

    def sums(x):
        dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
        u = torch.empty(len(x), 3, dtype=torch.float64, device="cuda")
        p = torch.empty(len(x), dtype=torch.float64, device="cuda")
        gpu_ctx.set_precision(core.FP64)
        F.ic2d_passive_sums(gpu_ctx, u, p, dev(x), dev(y), dev(y[:, 0].copy()), dev(a),
                            dev(np.zeros(len(y), np.uint8)), eps)
        gpu_ctx.synchronize()
        return np.c_[u.cpu().numpy(), p.cpu().numpy()]

    s = sums(x)
    assert np.isfinite(np.delete(s, 77, 0)).all()
    assert np.array_equal(s[77], sums(x[75:79])[2], equal_nan=True)


@pytest.mark.parametrize("collocated", [False, True])
def test_stream_function_alone(gpu_ctx, collocated):
    """Without the velocity: the same kernel over the same chunks, the same bits."""
    vx, fx, fa, fm = core.build_mesh(core.MESH_CUBED_SPHERE, 4, 1.0)
    y, a = fx[fm == 0], fa[fm == 0]
    x = y if collocated else vx
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    X, Y, Z, A, M = dev(x), dev(y), dev(y[:, 1].copy()), dev(a), dev(np.zeros(len(y), np.uint8))
    u = torch.empty(len(x), 3, dtype=torch.float64, device="cuda")
    p, q = (torch.empty(len(x), dtype=torch.float64, device="cuda") for _ in range(2))
    gpu_ctx.set_precision(core.FP64)
    for vel, psi in ((u, p), (None, q)):
        if collocated:
            F.ic2d_active_sums(gpu_ctx, vel, psi, Y, Z, A, M, 0.0, self_rule=1)
        else:
            F.ic2d_passive_sums(gpu_ctx, vel, psi, X, Y, Z, A, M, 0.0)
    gpu_ctx.synchronize()
    assert torch.isfinite(p).all() and torch.equal(p, q)
