"""2-D u8 images behind a cast to f32 on the tile kernel (the blur_png chain; 3
components from radius 8 on take the line passes): bit-exact against the oracle in reference rounding at the edges of tiles
(64 x 32) and of the word-staged interior, for 1 and 3 components, every output
type and sub-regions; explicit algorithms answer as before."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _case(gpu, arr, sigma, comps, rounding, out_dtype, request=None):
    dev = gpu.DeviceImage.from_host(gpu.Image(arr, components=comps))
    f = gpu.GaussianFilter(gpu.CastFilter(dev, gpu.F32), sigma, rounding=rounding)
    return f.generate_region(request or dev.region, out_dtype=out_dtype).download()


@pytest.mark.parametrize("shape", [(1, 1), (3, 200), (33, 65), (31, 63), (64, 128), (70, 131), (129, 193)])
@pytest.mark.parametrize("comps", [1, 3])
@pytest.mark.parametrize("radius", [1, 2, 5, 8, 12])
def test_reference_rounding_bit_exact(gpu, shape, comps, radius):
    rng = np.random.default_rng(shape[1] * 5 + radius)
    arr = rng.integers(0, 256, shape + ((3,) if comps == 3 else ()), dtype=np.uint8)
    want = oracle.gaussian_f32(arr.astype(np.float32), radius / 3.0, comps=comps)
    got = _case(gpu, arr, radius / 3.0, comps, gpu.ROUND_REFERENCE, gpu.F32)
    tiles = radius < 8 or comps == 1
    assert gpu.last_kernel() == ("tile2d_u8_ref" if tiles else "per_axis_f32_ref"), gpu.last_kernel()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    u8 = _case(gpu, arr, radius / 3.0, comps, gpu.ROUND_REFERENCE, gpu.U8)
    assert np.array_equal(u8, np.clip(np.floor(want.astype(np.float64) + 0.5), 0, 255).astype(np.uint8))
    fma = _case(gpu, arr, radius / 3.0, comps, gpu.ROUND_FMA, gpu.F32)
    # two passes of 2r + 1 terms of at most 255, each at most 2^-24 off per term, on both sides
    assert np.abs(fma - want).max() <= 4 * (2 * radius + 2) * 2.0 ** -24 * 255


@pytest.mark.parametrize("comps", [1, 3])
def test_subregions_with_every_alignment(gpu, comps):
    rng = np.random.default_rng(3)
    arr = rng.integers(0, 256, (90, 211) + ((3,) if comps == 3 else ()), dtype=np.uint8)
    want = oracle.gaussian_f32(arr.astype(np.float32), 1.4, comps=comps)
    for x0 in range(9, 14):
        got = _case(gpu, arr, 1.4, comps, gpu.ROUND_REFERENCE, gpu.F32, gpu.Region((x0, 7), (150, 61)))
        assert np.array_equal(got.view(np.uint32), want[7:68, x0:x0 + 150].view(np.uint32)), x0


def test_explicit_algorithms_answer_as_before(gpu):
    arr = np.random.default_rng(4).integers(0, 256, (40, 50), dtype=np.uint8)
    dev = gpu.DeviceImage.from_host(gpu.Image(arr))
    src = gpu.CastFilter(dev, gpu.F32)
    with pytest.raises(gpu.ItkgError):
        gpu.GaussianFilter(src, 1.0, algorithm=gpu.ALGO_FUSED).generate_region(dev.region)
    per_axis = gpu.GaussianFilter(src, 1.0, algorithm=gpu.ALGO_PER_AXIS).generate_region(dev.region).download()
    assert gpu.last_kernel() == "per_axis_f32_ref"
    auto = gpu.GaussianFilter(src, 1.0).generate_region(dev.region).download()
    assert np.array_equal(per_axis.view(np.uint32), auto.view(np.uint32))
