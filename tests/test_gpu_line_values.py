"""The line passes themselves (from radius 13 on always, from radius 8 on where
their grid has 128 blocks): infinities and NaN at the edges of runs (16
outputs) and strips (64 columns) reach the outputs whose windows hold them and
no other, in both roundings, and finite values are the oracle's bits."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _blocks(shape, comps=1):
    """Blocks of a pass along x, y and z (four runs of 16 a block, strips of 64 columns or lines)."""
    nz, ny, nx = shape
    runs = [-(-n // 16) for n in (nx, ny, nz)]
    groups = [-(-r // 4) for r in runs]
    return groups[0] * -(-nz * ny // 64), -(-nx // 64) * groups[1] * nz, -(-nx // 64) * groups[2] * ny


@pytest.mark.parametrize("shape,radii", [((96, 97, 130), (8, 9, 8)), ((96, 97, 130), (12, 8, 10)), ((40, 50, 70), (13, 13, 13)),
                                         ((33, 48, 129), (24, 13, 16)), ((17, 65, 64), (30, 14, 13))])
@pytest.mark.parametrize("rounding", [0, 1])
def test_non_finite_values(gpu, shape, radii, rounding):
    assert min(radii) >= 13 or min(_blocks(shape)) >= 128
    rng = np.random.default_rng(shape[2] + radii[0])
    arr = rng.standard_normal(shape).astype(np.float32)
    kernels = [rng.uniform(0.01, 0.1, 2 * r + 1) for r in radii]
    nz, ny, nx = shape
    for z, y, x, v in [(15, 16, 63, np.inf), (16, ny - 1, min(64, nx - 1), -np.inf), (0, 0, 0, np.nan), (nz - 1, ny // 2, nx - 1, np.inf)]:
        one = arr.copy()
        one[z, y, x] = v
        dev = gpu.DeviceImage.from_host(gpu.Image(one))
        got = gpu.SeparableFilter(dev, kernels, rounding=rounding, algorithm=gpu.ALGO_PER_AXIS).generate_region(dev.region).download()
        want = oracle.separable_f32(one, kernels, 1)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
        ok = np.isfinite(want)
        if rounding == gpu.ROUND_REFERENCE:
            assert np.array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))
        else:  # each of a pass's terms is rounded once, 2^-24 of the running sum at most, on both sides
            bound = np.prod([np.abs(k).sum() for k in kernels]) * np.abs(arr).max()
            tol = 2.0 ** -23 * sum(len(k) + 1 for k in kernels) * bound
            assert ok.any() and np.abs(got[ok].astype(np.float64) - want[ok]).max() <= tol
