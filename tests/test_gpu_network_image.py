"""lpm_farfield_grad is the gradient of the weights that lpm_farfield_get_weights
returns, also after a training run that failed (here: more samples than the device
holds, refused at their allocation) has reset them."""
import numpy as np
import pytest

from lpm_gb300 import core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fresh", [False, True])
def test_gradient_after_failed_training(gpu_ctx, fresh):
    from lpm_gb300.farfield import NNORM, NPARAM, FarField

    rng = np.random.default_rng(2)
    norm = np.zeros(NNORM, np.float32)
    norm[48:97] = 1.0
    ff, other = FarField(ctx=gpu_ctx), FarField(ctx=gpu_ctx)
    if not fresh:
        ff.set_weights(rng.uniform(-0.1, 0.1, NPARAM).astype(np.float32), norm)
    with pytest.raises(core.LpmError):
        ff.train(nsamples=2**31 - 1)
    other.set_weights(*ff.get_weights())
    x = rng.normal(size=(1280, 48)).astype(np.float32)
    y = rng.normal(size=(1280, 3)).astype(np.float32)
    assert np.array_equal(ff.grad(x, y), other.grad(x, y))
