"""lpm_farfield_grad reports a bounded device-side wait that gave up and then leaves
the caller's array as it was."""
import ctypes as C

import numpy as np
import pytest

from lpm_gb300 import core

pytestmark = pytest.mark.gpu


def test_no_gradient_after_a_timeout(gpu_ctx):
    from lpm_gb300.farfield import NNORM, NPARAM, FarField

    rng = np.random.default_rng(1)
    ff = FarField(ctx=gpu_ctx)
    norm = np.zeros(NNORM, np.float32)
    norm[48:97] = 1.0
    ff.set_weights(rng.uniform(-0.1, 0.1, NPARAM).astype(np.float32), norm)
    x, y = rng.normal(size=(640, 48)).astype(np.float32), rng.normal(size=(640, 3)).astype(np.float32)
    g = np.full(NPARAM, 7.0, np.float32)
    L = core.lib()
    assert L.lpm_wait_selftest(gpu_ctx.handle, 512) == core.LPM_OK
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert L.lpm_farfield_grad(ff._h, p(x), p(y), 640, p(g)) == core.LPM_ERR_TIMEOUT
    assert (g == 7.0).all()
    assert L.lpm_context_synchronize(gpu_ctx.handle) == core.LPM_OK
    assert L.lpm_farfield_grad(ff._h, p(x), p(y), 640, p(g)) == core.LPM_OK
    assert np.array_equal(g, ff.grad(x, y))
