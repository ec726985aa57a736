"""The line passes (radius 8 and above) on requests inside a longer image: the
last run of a request holds fewer outputs than a thread makes, and the source
ends at the request's last tap.  Bit-exact against the oracle from input
buffers that cover exactly the input region, for pieces of a streamed image
and for host buffers."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _same(got, want):
    return np.array_equal(got.view(np.uint32), want.view(np.uint32))


def _crop(a, region, within):
    sl = tuple(slice(region.index[d] - within.index[d], region.index[d] - within.index[d] + region.size[d])
               for d in reversed(range(region.dim)))
    return np.ascontiguousarray(a[sl])


def _tight(gpu, arr, kernels, requested, index):
    """The filter over a device buffer of exactly the request's input region."""
    full = gpu.Image(arr, index=index)
    need = gpu.SeparableFilter(full, kernels).input_region_for_output(requested)

    class Source(gpu.DeviceImage):
        def largest_region(self):
            return full.region

    dev = Source(need)
    dev.upload(_crop(arr, need, full.region))
    f = gpu.SeparableFilter(dev, kernels, algorithm=gpu.ALGO_PER_AXIS)
    return f.generate_region(requested).download()


# extents of 1, 15, 16 and 17 past whole runs, at the image's edges and inside
@pytest.mark.parametrize("shape,requested,radii", [
    ((900,), ((300,), (17,)), (24,)), ((900,), ((0,), (65,)), (13,)), ((300,), ((283,), (17,)), (60,)),
    ((230, 310), ((40, 33), (129, 31)), (24, 13)), ((230, 310), ((0, 100), (80, 65)), (8, 9)),
    ((90, 100, 110), ((20, 30, 35), (33, 47, 17)), (13, 24, 15)),
    ((90, 100, 110), ((70, 64, 0), (40, 36, 49)), (24, 13, 24)),
    ((70, 80, 200), ((30, 20, 25), (129, 16, 15)), (13, 9, 8)),
    ((60, 61, 300), ((101, 11, 21), (97, 33, 17)), (65, 8, 24))])
def test_requests_from_tight_buffers(gpu, shape, requested, radii):
    rng = np.random.default_rng(sum(shape))
    arr = rng.standard_normal(shape).astype(np.float32)
    index = tuple(-5 - 3 * d for d in range(len(shape)))
    at = tuple(i + o for i, o in zip(requested[0], index))
    kernels = [rng.uniform(-0.2, 0.3, 2 * r + 1) for r in radii]
    got = _tight(gpu, arr, kernels, gpu.Region(at, requested[1]), index)
    assert _same(got, oracle.separable_f32(arr, kernels, 1, index=index, requested=(at, requested[1])))


@pytest.mark.parametrize("shape,sigma", [((1500,), 5.0), ((230, 310), 4.5), ((75, 90, 97), 4.5), ((75, 60, 70), 8.0)])
def test_pieces_and_host_buffers(gpu, shape, sigma):
    arr = np.random.default_rng(shape[-1]).standard_normal(shape).astype(np.float32)
    want = oracle.gaussian_f32(arr, sigma)
    dev = gpu.DeviceImage.from_host(gpu.Image(arr))
    assert _same(gpu.stream_full(gpu.GaussianFilter(dev, sigma, algorithm=gpu.ALGO_PER_AXIS), 4).download(), want)
    host = gpu.GaussianFilter(gpu.Image(arr), sigma)
    assert _same(host.generate_region(host.source.region).data, want)


def test_staged_slabs(gpu):
    """A host image of several staging slabs (more than 8 MiB of output), radius 24."""
    arr = np.random.default_rng(4).standard_normal((150, 130, 128)).astype(np.float32)
    f = gpu.GaussianFilter(gpu.Image(arr), 8.0)
    assert _same(f.generate_region(f.source.region).data, oracle.gaussian_f32_mt(arr, 8.0))
