"""unsharp_front_f32 (itk-rs_gb300/csrc/unsharp.cuh), restated on the host in
tests/cpp/unsharp_front.c, never disagrees with the reference's f64 sequence
where it decides, and decides nearly every voxel of usual data."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_unsharp_front_rule(tmp_path):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("gcc not found")
    exe = str(tmp_path / "unsharp_front")
    subprocess.run([cc, "-O2", "-ffp-contract=off", os.path.join(HERE, "cpp", "unsharp_front.c"), "-o", exe, "-lm"],
                   check=True)
    r = subprocess.run([exe, "3000000"], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0 and " 0 mismatches" in r.stdout, r.stdout + r.stderr
