"""The two-pass z kernels on rows that end in a partial quad (stored in quads but
for the last one): bit-exact in reference rounding and u8 pixel arithmetic,
within the fused multiply-adds' rounding otherwise, on both sides of the radii
where the kernel's form changes (6 / 7, 8 / 9), with nothing written past a row."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [1, 3, 31, 33, 34, 63])
@pytest.mark.parametrize("radius", [1, 6, 7, 8, 9, 12])
def test_ragged_rows(gpu, nx, radius):
    sigma = radius / 3.0
    shape = (2 * radius + 5, 7, nx)
    rng = np.random.default_rng(nx * 13 + radius)
    x = rng.standard_normal(shape).astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    # the output image is wider than the request: what lies beyond it stays
    whole = gpu.Region((0, 0, 0), (nx + 6, 7, shape[0]))
    want = oracle.gaussian_f32(x, sigma)
    for rounding in (gpu.ROUND_REFERENCE, gpu.ROUND_FMA):
        out = gpu.DeviceImage(whole)
        out.upload(np.full((shape[0], 7, nx + 6), -7.0, np.float32))
        gpu.GaussianFilter(dev, sigma, rounding=rounding).generate_region(dev.region, out=out)
        assert gpu.last_kernel().startswith("z_pass_f32"), gpu.last_kernel()
        got = out.download()
        assert (got[..., nx:] == -7.0).all()
        if rounding == gpu.ROUND_REFERENCE:
            assert np.array_equal(got[..., :nx].view(np.uint32), want.view(np.uint32))
        else:
            # three passes of 2r + 1 terms, each at most 2^-24 off per term, on both sides
            assert np.abs(got[..., :nx] - want).max() <= 6 * (2 * radius + 2) * 2.0 ** -24 * np.abs(x).max()


@pytest.mark.parametrize("nx", [1, 15, 34, 63, 64])
@pytest.mark.parametrize("radius", [1, 6, 7, 9, 12])
def test_u8_ragged_rows(gpu, nx, radius):
    sigma = radius / 3.0
    x = np.random.default_rng(nx + radius).integers(0, 256, (2 * radius + 5, 9, nx), dtype=np.uint8)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    got = gpu.GaussianFilter(dev, sigma).generate_region(dev.region).download()
    assert gpu.last_kernel() == "z_pass_u8_pixel", gpu.last_kernel()
    assert np.array_equal(got, oracle.gaussian_u8(x, sigma))
