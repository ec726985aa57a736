"""The per-axis passes that walk runs of 16 outputs per thread (radius 8 and
above): bit-exact against the oracle in reference rounding, at the edges of
runs (16 outputs), strips (64 columns or lines) and block sizes, for every
input and output type, and with infinities and NaN kept to their windows."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _kernel(r, seed):
    return np.random.default_rng(seed).uniform(-0.2, 0.3, 2 * r + 1)


def _run(gpu, arr, kernels, rounding, components=1, out_dtype=None):
    dev = gpu.DeviceImage.from_host(gpu.Image(arr, components=components))
    src = dev if arr.dtype == np.float32 else gpu.CastFilter(dev, gpu.F32)
    f = gpu.SeparableFilter(src, kernels, rounding=rounding, algorithm=gpu.ALGO_PER_AXIS)
    return f.generate_region(dev.region, out_dtype=out_dtype).download()


def _want(arr, kernels, comps=1):
    return oracle.separable_f32(arr.astype(np.float32), kernels, 1, comps=comps)


# radius 8 is the shortest walk; 64 / 65 and 360 / 361 change the block size along x
@pytest.mark.parametrize("shape,radii", [((3, 5, 16), (8, 9, 8)), ((17, 16, 65), (8, 23, 13)),
                                         ((33, 47, 64), (24, 8, 16)), ((2, 31, 129), (64, 10, 12)),
                                         ((1, 66, 143), (65, 40, 8)), ((9, 2, 257), (360, 8, 97)),
                                         ((4, 3, 70), (361, 384, 384)), ((1, 1, 1), (8, 8, 8))])
def test_reference_rounding_bit_exact(gpu, shape, radii):
    arr = np.random.default_rng(shape[2]).standard_normal(shape).astype(np.float32)
    kernels = [_kernel(r, r + i) for i, r in enumerate(radii)]
    got = _run(gpu, arr, kernels, gpu.ROUND_REFERENCE)
    want = _want(arr, kernels)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    # fused multiply-adds: each of the K terms of a pass is rounded once (2^-24 of the running sum at most)
    fma = _run(gpu, arr, kernels, gpu.ROUND_FMA).astype(np.float64)
    bound = np.ones(())
    for k in kernels:
        bound = bound * np.abs(k).sum()
    tol = 2.0 ** -23 * sum(len(k) + 1 for k in kernels) * bound * np.abs(arr).max()
    assert np.abs(fma - want).max() <= tol


@pytest.mark.parametrize("components", [1, 2, 3])
@pytest.mark.parametrize("dtype", [np.float32, np.int16, np.uint8, np.float16])
def test_casts_and_components(gpu, dtype, components):
    if components > 1 and dtype != np.float32:
        pytest.skip("vector pixels are f32")
    shape = (37, 83) + ((components,) if components > 1 else ())
    rng = np.random.default_rng(5)
    arr = (rng.uniform(0, 200, shape)).astype(dtype)
    kernels = [np.full(2 * r + 1, 1.0 / (2 * r + 1)) for r in (9, 30)]
    want = _want(arr, kernels, comps=components)
    got = _run(gpu, arr, kernels, gpu.ROUND_REFERENCE, components)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    if components == 1:
        u8 = _run(gpu, arr, kernels, gpu.ROUND_REFERENCE, out_dtype=gpu.U8)
        assert np.array_equal(u8, np.clip(np.floor(want.astype(np.float64) + 0.5), 0, 255).astype(np.uint8))


def test_non_finite_values_stay_in_their_windows(gpu):
    arr = np.ones((40, 50, 70), np.float32)
    arr[20, 20, 30] = np.inf
    arr[5, 44, 66] = np.nan
    kernels = [np.full(17, 1.0 / 17)] * 3
    got = _run(gpu, arr, kernels, gpu.ROUND_REFERENCE)
    want = _want(arr, kernels)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))
