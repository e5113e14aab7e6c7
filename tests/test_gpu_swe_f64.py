"""The FP64 SWE sums at the sizes and inputs where the moment forms can go
wrong, against the FP64 oracle: tile and block remainders, PSE widths far below
the domain (exp underflows for most pairs), values around the table's seams, a
target exactly on a source with eps = 0 (the reference's non-finite values).

Tolerance 1e-12 of the largest value of an output, as the other FP64 tests:
targets and sources keep 0.02 apart where eps = 0."""
import math

import numpy as np
import pytest
import torch

from lpm_gb300 import functors as F

pytestmark = pytest.mark.gpu

TOL = 1e-12
COLS = {"du1dx1": 2, "du1dx2": 3, "du2dx1": 4, "du2dx2": 5, "laps": 6, "psi": 7, "phi": 8}


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _grid(n, shift, scale):
    """n points of a square lattice of spacing `scale`, moved by `shift` cells."""
    k = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    return scale * (np.stack([i % k, i // k], 1) + shift - k / 2)


def _close(got, ref):
    got = got.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
    f = np.isfinite(ref)
    return not f.any() or np.abs(got[f] - ref[f]).max() <= TOL * np.abs(ref[f]).max()


@pytest.mark.parametrize("ns,nt", [(1, 1), (63, 129), (64, 127), (65, 128), (1000, 333)])
@pytest.mark.parametrize("eps,pse,scale", [(0.0, 0.5, 0.2), (0.03, 0.02, 0.2), (0.1, 3.0, 1.0)])
@pytest.mark.parametrize("coincident", [False, True])
def test_plane(gpu_ctx, oracle, ns, nt, eps, pse, scale, coincident):
    from lpm_gb300 import core

    rng = np.random.default_rng(ns + nt)
    y, x = _grid(ns, 0.0, scale), _grid(nt, 0.37, scale)
    if coincident:
        x[nt // 2] = y[ns // 2]
    z, sg, a = rng.normal(size=ns), rng.normal(size=ns), np.full(ns, scale * scale)
    sx, sy, m = rng.normal(size=nt), rng.normal(size=ns), np.zeros(ns, np.uint8)
    gpu_ctx.set_precision(core.FP64)
    o = F.swe_plane_vertex_sums(gpu_ctx, _dev(x), _dev(sx), _dev(y), _dev(z), _dev(sg), _dev(a),
                                _dev(m), _dev(sy), eps, pse)
    gpu_ctx.synchronize()
    r = oracle.swe_plane_sums(x, sx, y, z, sg, a, m, sy, eps, pse)
    assert _close(o["u"], r[:, :2])
    for k, c in COLS.items():
        assert _close(o[k], r[:, c]), k


@pytest.mark.parametrize("scale", [1e-90, 1e-70, 1.0, 1e70, 1e75])
@pytest.mark.parametrize("eps", [0.0, 1e-9, 0.05, 3.0, 1e4])
def test_plane_scales(gpu_ctx, oracle, scale, eps):
    """Positions around the ends of the fixed-point range, eps from far below to far
    above the distances, pairs on an axis, close together and (eps > 0) coincident."""
    from lpm_gb300 import core

    rng = np.random.default_rng(7)
    n = 200
    x, y = rng.normal(size=(n, 2)), rng.normal(size=(n, 2))
    x[:40, 1] = y[:40, 1] = 0.0
    x[50] = y[60] + 1e-6
    if eps > 0:
        x[70] = y[80]
    x, y, eps, pse = x * scale, y * scale, eps * scale, 0.5 * scale
    z, sg, a = rng.normal(size=n), rng.normal(size=n), rng.uniform(0.5, 1.0, n)
    sx, sy, m = rng.normal(size=n), rng.normal(size=n), np.zeros(n, np.uint8)
    gpu_ctx.set_precision(core.FP64)
    o = F.swe_plane_vertex_sums(gpu_ctx, _dev(x), _dev(sx), _dev(y), _dev(z), _dev(sg), _dev(a),
                                _dev(m), _dev(sy), eps, pse)
    gpu_ctx.synchronize()
    r = oracle.swe_plane_sums(x, sx, y, z, sg, a, m, sy, eps, pse)
    assert _close(o["u"], r[:, :2])
    for k in ("psi", "phi"):
        assert _close(o[k], r[:, COLS[k]]), k
    if abs(math.log10(scale)) < 74:  # beyond, the oracle's pi R^2 leaves the normal range
        for k in ("du1dx1", "du1dx2", "du2dx1", "du2dx2", "laps"):
            assert _close(o[k], r[:, COLS[k]]), k


@pytest.mark.parametrize("ns,nt", [(1, 1), (63, 129), (64, 127), (65, 128), (700, 260)])
@pytest.mark.parametrize("eps", [0.05, 0.4])
def test_sphere(gpu_ctx, oracle, ns, nt, eps):
    from lpm_gb300 import core

    rng = np.random.default_rng(ns + nt)
    unit = lambda p: p / np.linalg.norm(p, axis=1, keepdims=True)
    y, x = unit(rng.normal(size=(ns, 3))), unit(rng.normal(size=(nt, 3)))
    z, sg, a = rng.normal(size=ns), rng.normal(size=ns), np.full(ns, 0.02)
    m = np.zeros(ns, np.uint8)
    gpu_ctx.set_precision(core.FP64)
    o = F.swe_sphere_vertex_sums(gpu_ctx, _dev(x), _dev(y), _dev(z), _dev(sg), _dev(a), _dev(m), eps,
                                 want_grad=True)
    gpu_ctx.synchronize()
    r = oracle.swe_sphere_sums(x, y, z, sg, a, m, eps)
    assert _close(o["u"], r[:, :3]) and _close(o["grad"], r[:, 3:])
