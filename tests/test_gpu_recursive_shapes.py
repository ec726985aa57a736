"""The recursive Gaussian on the shapes and buffers its line passes could trip
over: an axis beyond 2^30 samples, images a few columns wide (scratch rows),
and outputs that overlap the input elsewhere than voxel on voxel."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_an_axis_of_2_to_the_30(gpu):
    """2^30 columns of two u8 rows, filtered along y (every column stands alone)."""
    nx, L = 1 << 30, gpu._abi.lib()
    part = np.random.default_rng(0).integers(0, 256, (2, 4096), dtype=np.uint8)
    dev = gpu.DeviceImage(gpu.Region((0, 0), (nx, 2)), gpu.U8)
    for x0 in (0, nx - 4096):  # the two ends; what lies between is whatever the memory held
        for y in (0, 1):
            row = np.ascontiguousarray(part[y])
            gpu._abi.check(L.itkg_memcpy(ctypes.c_void_p(dev.c.data + y * dev.c.pitch[1] + x0), row.ctypes.data, row.nbytes, 0, None))
    gpu._abi.check(L.itkg_stream_synchronize(None))
    out = gpu.RecursiveGaussianAxisFilter(dev, 2.0, 1).generate_region(dev.region)
    want = oracle.from_f64_u8(oracle.recursive_gaussian_f64(part, 2.0, axis=1))
    for x0 in (0, nx - 4096):
        got = np.empty((2, 4096), np.uint8)
        for y in (0, 1):
            gpu._abi.check(L.itkg_memcpy(got[y].ctypes.data, ctypes.c_void_p(out.c.data + y * out.c.pitch[1] + x0), 4096, 1, None))
        gpu._abi.check(L.itkg_stream_synchronize(None))
        assert np.array_equal(got, want)


@pytest.mark.parametrize("nx", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("axis", [None, 0, 1])
def test_narrow_images(gpu, nx, axis):
    x = np.random.default_rng(nx).standard_normal((9, 50, nx)).astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    got = gpu.RecursiveGaussianFilter(dev, 1.7, axis=axis).generate_region(dev.region).download()
    want = oracle.recursive_gaussian_f32(x, 1.7, axis=-1 if axis is None else axis)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


ONE_COLUMN = """
import sys
sys.path.insert(0, {root!r} + "/itk-rs_gb300")
import itkg, torch
n = 1 << 12
region = itkg.Region((0, 0, 0), (1, 4, 4))
warm = itkg.DeviceImage(region, itkg.U8)
itkg.RecursiveGaussianFilter(warm, 2.0).generate_region(region)
dev, free = itkg.DeviceImage(itkg.Region((0, 0, 0), (1, n, n)), itkg.U8), []
for i in range(2):
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
    out = itkg.RecursiveGaussianFilter(dev, 2.0).generate_region(region)
print(free[0] - free[1])
"""


def test_scratch_of_a_one_column_image(gpu):
    """8 bytes of scratch a sample, 128 MiB for 2^24, not rows of four (512 MiB)."""
    p = subprocess.run([sys.executable, "-c", ONE_COLUMN.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    assert int(p.stdout.split()[-1]) < 320 << 20, p.stdout


# (the last two: more lines than the device holds threads for, the output over lines of later blocks)
@pytest.mark.parametrize("shape,axis,shift", [((80, 64), 0, 0), ((80, 64), 0, 1), ((80, 64), 1, 0), ((80, 64), 1, 192),
                                              ((600000, 8), 0, 8 * 250000), ((6, 700000), 1, 300000)])
def test_output_over_the_input(gpu, shape, axis, shift):
    """One filtered axis, the output `shift` samples further on in the input's memory."""
    x = np.random.default_rng(shift).standard_normal(shape).astype(np.float32)
    big = gpu.DeviceImage(gpu.Region((0,), (x.size + shift,)))
    big.upload(np.concatenate([x.ravel(), np.zeros(shift, np.float32)]))
    L, im = gpu._abi.lib(), gpu.Image(x)
    src, dst = im.to_c(), im.to_c()
    for c, off in ((src, 0), (dst, 4 * shift)):
        c.location, c.data = gpu._abi.DEVICE, big.c.data + off
    f = gpu.RecursiveGaussianFilter(im, 2.0, axis=axis)
    reg, prm = im.region.to_c(), f.params()
    gpu._abi.check(L.itkg_recursive_gaussian_generate_region(ctypes.byref(src), ctypes.byref(reg), ctypes.byref(reg),
                                                             ctypes.byref(prm), ctypes.byref(dst), None))
    got = big.download()[shift:].reshape(shape)
    assert np.array_equal(got.view(np.uint32), oracle.recursive_gaussian_f32(x, 2.0, axis=axis).view(np.uint32))


@pytest.mark.parametrize("shape,axis", [((257,), None), ((4,), 0), ((300, 128), 1), ((300, 129), 1), ((128, 71), 0), ((129, 71), 0),
                                        ((8, 16, 40), 0), ((8, 17, 40), 0), ((61, 8, 16), 2)])
@pytest.mark.parametrize("dtype", [np.float32, np.uint8, np.int16])
def test_few_lines_of_one_axis(gpu, shape, axis, dtype):
    """Both sides of the 128 lines up to which the conversions run apart; whole images and sub-regions."""
    rng = np.random.default_rng(sum(shape))
    x = rng.integers(0, 256, shape).astype(dtype) if dtype != np.float32 else rng.standard_normal(shape).astype(dtype)
    f64 = oracle.recursive_gaussian_f64(x.astype(np.float64), 1.9, axis=-1 if axis is None else axis)
    want = oracle.from_f64_u8(f64) if dtype == np.uint8 else f64.astype(np.float32)
    dev = gpu.DeviceImage.from_host(gpu.Image(x))
    f = gpu.RecursiveGaussianFilter(dev, 1.9, axis=axis)
    for at, size in [((0,) * x.ndim, tuple(reversed(shape))), (tuple(n // 3 for n in reversed(shape)), tuple((n + 3) // 4 for n in reversed(shape)))]:
        got = f.generate_region(gpu.Region(at, size)).download()
        sl = tuple(slice(at[d], at[d] + size[d]) for d in reversed(range(x.ndim)))
        assert got.dtype == want.dtype and np.array_equal(got.view(np.uint8), np.ascontiguousarray(want[sl]).view(np.uint8))
