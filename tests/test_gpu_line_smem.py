"""The line pass along x at radii where its shared memory passes 48 KB, static
part included: as a process's first launch of the kernel, and from threads
whose radii differ."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIRST = """
import sys
sys.path[:0] = [{root!r} + "/itk-rs_gb300", {root!r} + "/oracle"]
import itkg, numpy as np, oracle
x = np.random.default_rng({r}).standard_normal((3, {nx})).astype(np.float32)
k = [np.random.default_rng(1).uniform(-0.2, 0.3, 2 * {r} + 1), np.ones(1)]
d = itkg.DeviceImage.from_host(itkg.Image(x))
got = itkg.SeparableFilter(d, k, algorithm=itkg.ALGO_PER_AXIS).generate_region(d.region).download()
assert np.array_equal(got.view(np.uint32), oracle.separable_f32(x, k, 1).view(np.uint32))
"""


# 4, 3, 2 and 1 warps per block: the dynamic part is just under 48 KB
@pytest.mark.parametrize("r,nx", [(60, 64), (61, 130), (68, 48), (76, 32), (84, 16)])
def test_first_launch_of_a_process(gpu, r, nx):
    p = subprocess.run([sys.executable, "-c", FIRST.format(root=ROOT, r=r, nx=nx)], capture_output=True, text=True,
                       timeout=120)
    assert p.returncode == 0, p.stderr


def test_threads_of_different_radii(gpu):
    x = np.random.default_rng(0).standard_normal((2, 400)).astype(np.float32)
    jobs = {r: [np.random.default_rng(r).uniform(-0.2, 0.3, 2 * r + 1), np.ones(1)] for r in (61, 70, 150, 300)}
    want = {r: oracle.separable_f32(x, k, 1) for r, k in jobs.items()}
    bad = []

    def work(r):
        try:
            d = gpu.DeviceImage.from_host(gpu.Image(x))
            f = gpu.SeparableFilter(d, jobs[r], algorithm=gpu.ALGO_PER_AXIS)
            for _ in range(200):
                out = f.generate_region(d.region)
            if not np.array_equal(out.download().view(np.uint32), want[r].view(np.uint32)):
                bad.append((r, "values"))
        except Exception as e:  # noqa: BLE001
            bad.append((r, str(e)))

    threads = [threading.Thread(target=work, args=(r,)) for r in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
