"""The recursive Gaussian on the shapes and buffers its line passes could trip
over: an axis beyond 2^30 samples, images a few columns wide (scratch rows),
and outputs that overlap the input elsewhere than voxel on voxel."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


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
