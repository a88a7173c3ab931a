"""Kernels that start before the previous kernel of their stream has ended, read
as sources (CPU).

What such a kernel loads may still be written during its lifetime, so it must not
use non-coherent loads (ld.global.nc: __ldg, or a load that the compiler turns
into one because the pointer is const __restrict__): these are defined only for
memory that nobody writes while the kernel runs, and the compiler may move them
ahead of the wait for the previous kernel.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chime-x_b200",
                    "csrc")


def _balanced(src, at, opening, closing):
    """The text from the bracket at `at` to its partner."""
    depth = 0
    for i in range(at, len(src)):
        depth += {opening: 1, closing: -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i + 1]
    raise AssertionError("unbalanced source")


def kernels():
    """{name: (parameters, body)} of every __global__ function."""
    found = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s*(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", src):
            params = _balanced(src, m.end() - 1, "(", ")")
            body = _balanced(src, src.index("{", m.end() - 1 + len(params)), "{", "}")
            found[m.group(1)] = (params, body)
    return found


KERNELS = kernels()
OVERLAPPED = sorted(n for n, (_, body) in KERNELS.items() if "pdl_wait(" in body)


def test_the_overlapped_kernels_are_found():
    assert {"tc_pair_kernel", "tc_small_kernel", "zero_kernel", "offset_accumulate_kernel",
            "preseed_kernel", "blocks_to_triangle_kernel", "blocks_to_full_kernel",
            "frame_copy_kernel", "noalloc_tables_kernel"} <= set(OVERLAPPED)


def test_every_overlapped_launch_waits():
    """launch_pdl and the programmatic attribute are used for these kernels only."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"launch_pdl\(\s*(\w+)", src):
            assert m.group(1) in OVERLAPPED, (path, m.group(1))


@pytest.mark.parametrize("name", OVERLAPPED)
def test_no_non_coherent_loads(name):
    params, body = KERNELS[name]
    assert "__restrict__" not in params, "loads through it may become non-coherent"
    assert not re.search(r"__ldg\(|ld\.global\.nc|__restrict__", body)
