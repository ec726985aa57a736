"""UnsharpMaskFilter in reference rounding from 2^22 voxels on (blur into the
output image, point-wise step in place): bit-exact against the oracle on both
sides of that size, with ragged rows, amounts that are f32 (ties decided in
f32) or not (f64), and an output that is the input image."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _same(got, want):
    return np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("shape", [(128, 128, 256), (128, 128, 255), (67, 89, 90), (61, 230, 333), (2049, 2050), (725, 727)])
@pytest.mark.parametrize("amount", [0.5, 0.37])
def test_bit_exact(gpu, shape, amount):
    x = np.random.default_rng(shape[-1]).standard_normal(shape).astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    got = gpu.UnsharpMaskFilter(dev, 1.2, amount, 0.05).generate_region(dev.region).download()
    assert _same(got, oracle.unsharp_mask(x, 1.2, amount, 0.05))


def test_output_is_the_input(gpu):
    x = np.random.default_rng(9).standard_normal((130, 180, 184)).astype(np.float32)
    want = oracle.unsharp_mask(x, 1.0, 0.5, 0.0)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    gpu.UnsharpMaskFilter(dev, 1.0, 0.5).generate_region(dev.region, out=dev)
    assert _same(dev.download(), want)
