"""lpm_farfield_grad at its smallest sizes, where the gradient is larger than the
rows it is made of: against the same rows repeated eight times (the loss scale
2 / n is an eighth exactly, so every tile's BF16 roundings and FP32 gradients are
the same but for that factor, and only FP64 sums in another order and the last
rounding to FP32 differ: 1e-6 of the largest entry), and against itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 256, 384, 512, 640, 1152])
def test_gradient_of_few_rows(gpu_ctx, n):
    from lpm_gb300.farfield import NNORM, NPARAM, FarField

    rng = np.random.default_rng(n)
    ff = FarField(ctx=gpu_ctx)
    norm = np.zeros(NNORM, np.float32)
    norm[48:97] = 1.0
    ff.set_weights(rng.uniform(-0.1, 0.1, NPARAM).astype(np.float32), norm)
    x = rng.normal(size=(n, 48)).astype(np.float32)
    y = rng.normal(size=(n, 3)).astype(np.float32)
    ref = ff.grad(np.tile(x, (8, 1)), np.tile(y, (8, 1)))
    g = [ff.grad(x, y) for _ in range(8)]
    assert all(np.array_equal(g[0], a) for a in g[1:])
    assert np.abs(g[0] - ref).max() <= 1e-6 * np.abs(ref).max()
