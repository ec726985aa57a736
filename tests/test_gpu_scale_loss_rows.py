"""The multi-scale loss on rows that are no multiple of 4 floats: on the two-pass
kernels from 2^14 voxels on, per axis below; loss, dL/dx and dL/dsigma_l against
FP64 numpy with the bounds of tests/test_gpu_vjp.py."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kernels", [((26, 27, 25), "two_pass"), ((25, 26, 23), "per_axis"),
                                           ((40, 13, 47), "two_pass"), ((30, 31, 1), "per_axis"),
                                           ((130, 127, 2), "two_pass")])
def test_ragged_rows_match_fp64(gpu, shape, kernels):
    rng = np.random.default_rng(sum(shape))
    x, t = rng.random(shape).astype(np.float32), rng.random(shape).astype(np.float32)
    sigmas = [0.7, 1.9, 3.8]
    dx, dt = (gpu.DeviceImage.from_host(gpu.Image(v)) for v in (x, t))
    loss, xbar, sb = gpu.scale_stack_loss_vjp(dx, dt, sigmas)
    assert gpu.last_kernel() == f"scale_stack_loss_vjp_{kernels}_f32", gpu.last_kernel()
    x64, t64 = x.astype(np.float64), t.astype(np.float64)
    want_loss, want_x = 0.0, np.zeros(shape)
    for s, g in zip(sigmas, sb):
        radii = [int(np.ceil(3 * s))] * 3
        d = oracle.gaussian_whole_f64(x64, s, radii=radii) - t64
        want_loss += float((d * d).sum())
        want_x += oracle.gaussian_adjoint_f64(2 * d, s, radii=radii)
        want = float((2 * d * oracle.gaussian_dsigma_f64(x64, s, radii=radii)).sum())
        assert abs(g - want) <= 1e-4 * max(1.0, abs(want)), (s, g, want)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.abs(xbar.download().astype(np.float64) - want_x).max() <= 1e-5 * np.abs(want_x).max()
