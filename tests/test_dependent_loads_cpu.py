"""Kernels that start before the stream's previous kernel has ended
(griddepcontrol.wait) read global memory with ordinary loads only: read-only
loads (__ldg, ld.global.nc) ask for memory that nothing writes while the
kernel runs, and the previous kernel may still be writing it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "itk-rs_gb300", "csrc")


def _kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        start = text.index("{", text.index(")", text.index("k_", m.start())))
        name = re.search(r"\bk_\w+", text[m.start():start]).group(0)
        depth, i = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield name, text[start:i]


def test_no_read_only_loads_behind_a_dependent_launch():
    dependent, bad = set(), []
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for name, body in _kernels(text):
            if "griddepcontrol.wait" in body or "pdl_begin" in body:
                dependent.add(name)
                if re.search(r"__ldg|ld\.global\.nc|__restrict__", body):
                    bad.append(name)
    assert {"k_lines_yz", "k_lines_x", "k_xy_vjp", "k_z_adj2", "k_xy_pass", "k_z_pass", "k_unsharp_quads", "k_sqerr_q",
            "k_sum_partials"} <= dependent
    assert not bad, bad
