"""2-D u8 images behind a cast, filtered into the image they come from."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,sigma", [((300, 400), 1.5), ((517, 700), 3.0), ((90, 130, 3), 2.0), ((1200, 1100), 2.0)])
def test_output_is_the_input(gpu, shape, sigma):
    comps = 3 if len(shape) == 3 else 1
    x = np.random.default_rng(shape[0]).integers(0, 256, shape, dtype=np.uint8)
    want = oracle.cast_f32_to_u8(oracle.gaussian_f32(x.astype(np.float32), sigma, comps=comps))
    dev = gpu.DeviceImage.from_host(gpu.Image(x, components=comps))
    f = gpu.GaussianFilter(gpu.CastFilter(dev, gpu.F32), sigma)
    f.generate_region(dev.region, out_dtype=gpu.U8, out=dev)
    assert np.array_equal(dev.download(), want)
