"""lpm_bve_rk4_kernel_shape of FP64 steppers: the threads and targets per thread of
the kernel that the plan holds.  4,096 targets by 1,024 sources and more run the split
sums (64 threads, one target each, capped for 8 CTAs per SM); grids of less than two
waves of the tiled kernels the one-target-per-thread form (64, 1); the others 128
threads of two targets."""
import pytest

from lpm_gb300 import core
from lpm_gb300.bve import BVERK4, BVESphere, rossby_haurwitz_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,level,shape", [
    (core.FP64, 4, (64, 1, 8)), (core.FP64, 2, (64, 1, 0)),
    (core.FP64_EXACT, 2, (64, 1, 0)), (core.FP64_EXACT, 5, (128, 2, 0)),
    (core.FP64_CHORD, 2, (64, 1, 0)), (core.FP64_CHORD, 5, (128, 2, 0))])
def test_fp64_kernel_shape(gpu_ctx, precision, level, shape):
    sph = BVESphere(level, ctx=gpu_ctx)
    sph.init_vorticity(core.IC_RH54, rossby_haurwitz_params())
    gpu_ctx.set_precision(core.FP64)
    sph.init_velocity()
    st = BVERK4(0.001, sph, precision=precision)
    st.advance_timestep(sph)
    gpu_ctx.synchronize()
    assert st.kernel_shape() == shape
    st.close()
