"""The octree and target blocks built on the device against the host build
(lpm_octree_stats): the same number of cells and blocks, and the far-field sum
over them against the direct sum, at the sizes where the build can go wrong
(one point, leaf and block limits, tile remainders), with coincident points down
to the last level, and when a far field is reused for larger and smaller problems.

Tolerance: theta 0.3 expansions are within 1e-3 of the largest velocity (the
truncation (h / D)^5 of cells with at least 32 points); with fewer than 32
sources per accepted cell the sum is the FP32 direct one, within 1e-5."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(rng, n):
    x = rng.normal(size=(n, 3))
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _check(ctx, oracle, ff, x, y, z, leaf_max, eps=0.1):
    from lpm_gb300.farfield import octree_stats

    n = len(y)
    a, m = np.full(n, 4 * np.pi / n), np.zeros(n, np.uint8)
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()
    u = torch.zeros(len(x), 3, dtype=torch.float64, device="cuda")
    ff.velocity(u, dev(x), dev(y), dev(z), dev(a), dev(m), eps)
    ctx.synchronize()
    want, got = octree_stats(y, x, leaf_max), ff.stats()
    assert (got["cells"], got["target_blocks"]) == (want["cells"], want["blocks"])
    with oracle.chord_form():
        ur, _ = oracle.ic2d_passive_sums(x, y, z, a, m, eps)
    return np.abs(u.cpu().numpy() - ur).max() / np.abs(ur).max()


@pytest.mark.parametrize("ns,nt,leaf_max", [(1, 1, 64), (64, 128, 64), (65, 129, 64), (9, 1025, 1),
                                            (1023, 2049, 64), (1025, 1024, 17), (5000, 7001, 64)])
def test_sizes(gpu_ctx, oracle, ns, nt, leaf_max):
    from lpm_gb300.farfield import FarField

    rng = np.random.default_rng(ns)
    ff = FarField(theta=0.3, leaf_max=leaf_max, ctx=gpu_ctx)
    err = _check(gpu_ctx, oracle, ff, _points(rng, nt), _points(rng, ns), rng.normal(size=ns), leaf_max)
    assert err < 1e-3


def test_coincident_points(gpu_ctx, oracle):
    """More equal points than a leaf or a block holds: split to the last level,
    then cut into blocks."""
    from lpm_gb300.farfield import FarField

    rng = np.random.default_rng(2)
    y, x = _points(rng, 1500), _points(rng, 1500)
    y[100:400] = y[100]
    x[200:700] = x[200]
    ff = FarField(theta=0.3, ctx=gpu_ctx)
    assert _check(gpu_ctx, oracle, ff, x, y, rng.normal(size=1500), 64) < 1e-3


def test_reuse_grows_and_shrinks(gpu_ctx, oracle):
    """One far field over problems of changing size: its buffers are kept, the
    values are those of a new one."""
    from lpm_gb300.farfield import FarField

    rng = np.random.default_rng(4)
    ff = FarField(theta=0.3, ctx=gpu_ctx)
    for n in (700, 4000, 90, 4000):
        y, x, z = _points(rng, n), _points(rng, n // 2), rng.normal(size=n)
        a = _check(gpu_ctx, oracle, ff, x, y, z, 64)
        b = _check(gpu_ctx, oracle, FarField(theta=0.3, ctx=gpu_ctx), x, y, z, 64)
        assert a == b and a < 1e-3


@pytest.mark.parametrize("theta", [0.05, 0.12])
def test_long_lists(gpu_ctx, oracle, theta):
    """Interaction lists longer than a warp's ordered list (2,048 cells): those
    blocks walk serially; leaves of one point make the lists long.  Every pair is
    then a near one or an accepted cell of fewer than 32 points: the FP32 direct
    sum, within 1e-5."""
    from lpm_gb300.farfield import FarField

    rng = np.random.default_rng(6)
    ff = FarField(theta=theta, leaf_max=1, rho_min=0.0, ctx=gpu_ctx)
    err = _check(gpu_ctx, oracle, ff, _points(rng, 300), _points(rng, 3500), rng.normal(size=3500), 1)
    assert err < (1e-5 if theta < 0.1 else 1e-3)
