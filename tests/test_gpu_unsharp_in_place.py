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


@pytest.mark.parametrize("shape", [(301, 403), (65, 256, 257)])
def test_a_call_without_memory_leaves_the_output(gpu, shape):
    """Whichever of the call's scratch allocations fails, the output keeps what it held."""
    from itkg import _abi
    L = _abi.lib()
    x = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    old = np.random.default_rng(2).standard_normal(shape).astype(np.float32)
    dev, out = gpu.DeviceImage.from_host(gpu.Image(x)), gpu.DeviceImage.from_host(gpu.Image(old))
    f = gpu.UnsharpMaskFilter(dev, 1.2, 0.37, 0.02)
    failed = 0
    for after in range(8):
        L.itkg_debug_fail_scratch_alloc(after)
        try:
            f.generate_region(dev.region, out=out)
            break
        except _abi.ItkgError as e:
            assert e.status == _abi.ERROR_OUT_OF_MEMORY
            failed += 1
        finally:
            L.itkg_debug_fail_scratch_alloc(-1)
        assert np.array_equal(out.download().view(np.uint32), old.view(np.uint32)), after
    assert failed < 8  # (a 2-D call takes no scratch)
    assert np.array_equal(out.download().view(np.uint32), oracle.unsharp_mask(x, 1.2, 0.37, 0.02).view(np.uint32))


def test_a_small_call_is_three_launches(gpu):
    """x-y, z and point-wise kernel, also for an amount that is no f32."""
    x = np.random.default_rng(3).standard_normal((47, 46, 45)).astype(np.float32)
    dev, out = gpu.DeviceImage.from_host(gpu.Image(x)), gpu.DeviceImage.from_host(gpu.Image(x))
    n0 = gpu._abi.lib().itkg_launch_counter()
    gpu.UnsharpMaskFilter(dev, 1.2, 0.37, 0.02).generate_region(dev.region, out=out)
    assert gpu._abi.lib().itkg_launch_counter() - n0 == 3
    assert np.array_equal(out.download().view(np.uint32), oracle.unsharp_mask(x, 1.2, 0.37, 0.02).view(np.uint32))


@pytest.mark.parametrize("at,size", [((1, 3), (251, 64)), ((4, 0), (200, 90)), ((3, 2, 1), (61, 50, 20))])
def test_requests_off_the_quads(gpu, at, size):
    """Requests that start between the output image's quads."""
    shape = (100, 260) if len(at) == 2 else (30, 60, 70)
    x = np.random.default_rng(size[0]).standard_normal(shape).astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    out = gpu.DeviceImage.from_host(gpu.Image(np.zeros(shape, np.float32)))
    gpu.UnsharpMaskFilter(dev, 1.1, 0.37, 0.02).generate_region(gpu.Region(at, size), out=out)
    want = np.zeros(shape, np.float32)
    sl = tuple(slice(at[d], at[d] + size[d]) for d in reversed(range(len(at))))
    want[sl] = oracle.unsharp_mask(x, 1.1, 0.37, 0.02, requested=(at, size))
    assert np.array_equal(out.download().view(np.uint32), want.view(np.uint32))


def test_rows_off_the_quads_take_a_blur_image(gpu):
    """An output whose quads lie off the request's takes one scratch image more than one where they do not."""
    x = np.random.default_rng(3).standard_normal((47, 46, 45)).astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    f = gpu.UnsharpMaskFilter(dev, 1.2, 0.37, 0.02)
    req = gpu.Region((4, 0, 0), (37, 46, 47))
    L = gpu._abi.lib()
    allocs = []
    for x0 in (4, 3):
        out = gpu.DeviceImage(gpu.Region((x0, 0, 0), (41 - x0, 46, 47)))
        n0 = L.itkg_scratch_alloc_counter()
        f.generate_region(req, out=out)
        allocs.append(L.itkg_scratch_alloc_counter() - n0)
        want = oracle.unsharp_mask(x, 1.2, 0.37, 0.02, requested=(req.index, req.size))
        assert np.array_equal(out.download()[..., 4 - x0:].view(np.uint32), want.view(np.uint32))
    assert allocs[1] == allocs[0] + 1
