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
