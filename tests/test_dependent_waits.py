"""Kernels that may start under the kernel before them wait for it by dyb_grid_dep_wait (csrc/common.cuh), whose branch keeps __ldg and const __restrict__ loads behind
the wait; an asm statement alone does not.  Checked in the source: whether such a load moves is up to the compiler of the day."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynet_b200", "csrc")
# kernels that are only ever launched behind the whole of the kernel before them: dyb_launch with more than 96 KB of shared memory
ORDINARY = {"k_gemm_pair", "k_gemm_persist", "k_lstm_seq_bwd"}


def kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^;{]*\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield m.group(1), text[m.end():end]


def test_kernels_wait_by_the_helper():
    found = list(kernels())
    assert len(found) > 80 and ORDINARY <= {k for k, _ in found}
    assert {k for k, body in found if "dyb_grid_dep_" not in body} <= ORDINARY


def test_ordinary_kernels_are_not_launched_dependently():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            text = open(os.path.join(CSRC, name)).read()
            for k in ORDINARY:
                assert not re.search(r"dyb_launch_as\(\s*true,\s*%s\b" % k, text)
