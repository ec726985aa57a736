"""UnsharpMaskFilter with the input image as its output: bit-exact against the
oracle, in either form of the call (blur and step in one, or one after the
other), for amounts that are no f32 (voxels decided in f64 by a second
kernel) and for ones that are."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(150, 260), (301, 403), (2050, 2052), (30, 50, 61), (40, 64, 64), (130, 180, 184)])
@pytest.mark.parametrize("amount", [0.37, 0.1, 0.5])
def test_output_is_the_input(gpu, shape, amount):
    x = np.random.default_rng(shape[-1]).standard_normal(shape).astype(np.float32)
    want = oracle.unsharp_mask(x, 1.2, amount, 0.02)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    gpu.UnsharpMaskFilter(dev, 1.2, amount, 0.02).generate_region(dev.region, out=dev)
    assert np.array_equal(dev.download().view(np.uint32), want.view(np.uint32))
