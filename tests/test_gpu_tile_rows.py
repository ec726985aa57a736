"""Tile heights of the two-pass forward's x-y kernel: heights on both sides of
where 64-, 96- and 128-row tiles take over from each other, several tiles high
and with last tiles of a few rows, at radii with any of them (<= 8) and with 64
rows (9); the i16 and u8 forms too.  Reference rounding and u8 pixel arithmetic
are bit-exact, fused multiply-adds within their rounding."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [1, 31, 63, 64, 65, 95, 96, 97, 128, 129, 192, 193, 257, 288, 320])
@pytest.mark.parametrize("radius", [1, 3, 4, 6, 8, 9])
def test_heights(gpu, ny, radius):
    sigma = radius / 3.0
    shape = (radius + 2, ny, 41)
    x = np.random.default_rng(ny * 17 + radius).integers(-2000, 2000, shape).astype(np.int16)
    xf = x.astype(np.float32)
    want = oracle.gaussian_f32(xf, sigma)
    for img in (gpu.Image(xf), gpu.Image(x)):
        dev = gpu.DeviceImage.from_host(img)
        for rounding in (gpu.ROUND_REFERENCE, gpu.ROUND_FMA):
            out = gpu.DeviceImage(dev.region)
            gpu.GaussianFilter(dev, sigma, rounding=rounding).generate_region(dev.region, out=out)
            assert gpu.last_kernel().startswith("z_pass_f32"), gpu.last_kernel()
            got = out.download()
            if rounding == gpu.ROUND_REFERENCE:
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
            else:
                # three passes of 2r + 1 terms, each at most 2^-24 off per term, on both sides
                assert np.abs(got - want).max() <= 6 * (2 * radius + 2) * 2.0 ** -24 * np.abs(xf).max()


@pytest.mark.parametrize("ny", [31, 64, 96, 97, 192, 257, 320])
@pytest.mark.parametrize("radius", [1, 3, 4, 6, 8, 9])
def test_u8_heights(gpu, ny, radius):
    sigma = radius / 3.0
    x = np.random.default_rng(ny + radius).integers(0, 256, (radius + 2, ny, 41), dtype=np.uint8)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    got = gpu.GaussianFilter(dev, sigma).generate_region(dev.region).download()
    assert gpu.last_kernel() == "z_pass_u8_pixel", gpu.last_kernel()
    assert np.array_equal(got, oracle.gaussian_u8(x, sigma))
