"""The FP64 planar SWE sums at values that are not finite."""
import numpy as np
import pytest
import torch

from lpm_gb300 import core
from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu

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
