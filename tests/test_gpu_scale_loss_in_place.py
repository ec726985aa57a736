"""One level of the multi-scale loss with its gradient written over x."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(26, 27, 25), (40, 45, 47), (30, 32, 64)])
def test_gradient_over_x(gpu, shape):
    rng = np.random.default_rng(sum(shape))
    x, t = rng.random(shape).astype(np.float32), rng.random(shape).astype(np.float32)
    dx, dt = (gpu.DeviceImage.from_host(gpu.Image(v)) for v in (x, t))
    loss, xbar, sb = gpu.scale_stack_loss_vjp(dx, dt, [1.9])
    loss2, _, sb2 = gpu.scale_stack_loss_vjp(dx, dt, [1.9], xbar=dx)
    # apart and over x: at most the kernels' different order of sums
    assert abs(loss2 - loss) <= 1e-6 * abs(loss)
    assert abs(sb2[0] - sb[0]) <= 1e-4 * max(1.0, abs(sb[0]))
    want = xbar.download().astype(np.float64)
    assert np.abs(dx.download() - want).max() <= 1e-5 * np.abs(want).max()
