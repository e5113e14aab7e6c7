"""lpm_farfield_grad over more tiles than one slab of partial gradients holds:
the gradient of 512 tiles is the mean of its halves' gradients (the loss scale
2 / n halves exactly, so every BF16 rounding is the same and only FP32 products
and FP64 sums in another order differ: 1e-6 of the largest entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [256, 257])
def test_gradient_over_slabs(gpu_ctx, tiles):
    from lpm_gb300.farfield import NNORM, NPARAM, FarField

    rng = np.random.default_rng(tiles)
    ff = FarField(ctx=gpu_ctx)
    norm = np.zeros(NNORM, np.float32)
    norm[48:97] = 1.0
    ff.set_weights(rng.uniform(-0.1, 0.1, NPARAM).astype(np.float32), norm)
    n = 128 * tiles
    x = rng.normal(size=(2 * n, 48)).astype(np.float32)
    y = rng.normal(size=(2 * n, 3)).astype(np.float32)
    g, a, b = ff.grad(x, y), ff.grad(x[:n], y[:n]), ff.grad(x[n:], y[n:])
    assert np.abs(g - 0.5 * (a + b)).max() <= 1e-6 * np.abs(g).max()
