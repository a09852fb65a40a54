"""Rows of the sort-and-pad step past 2^31: the header with the kernels' row arithmetic, compiled for
the host.  (A run at that size needs 26 GB; the arithmetic does not.)"""

import ctypes
import os
import subprocess

import pytest

from moe_bench_b200 import build as mb_build

MAX_ASSIGNMENTS = 2**31 - 4097  # the most the sort accepts


@pytest.fixture(scope="module")
def sorted_row(tmp_path_factory):
    d = tmp_path_factory.mktemp("align_row")
    src, lib = os.path.join(d, "row.cpp"), os.path.join(d, "row.so")
    with open(src, "w") as f:
        f.write('#include "align_row.h"\n'
                'extern "C" int64_t row(int block, int pad, int before) { return mb200::sorted_row(block, pad, before); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{mb_build.CSRC}", src, "-o", lib], check=True)
    fn = ctypes.CDLL(lib).row
    fn.restype, fn.argtypes = ctypes.c_int64, [ctypes.c_int32] * 3
    return fn


@pytest.mark.parametrize("experts", [1, 256, 1024])
@pytest.mark.parametrize("pad", [1, 16, 128, 1024])
def test_last_row_of_the_largest_sort(sorted_row, experts, pad):
    # the last expert gets all but one assignment of every other expert: the most padding ahead of it
    last = MAX_ASSIGNMENTS - (experts - 1)
    assert sorted_row(experts - 1, pad, last - 1) == (experts - 1) * pad + last - 1
    # and evenly spread: every segment a multiple of pad, plus one
    per = MAX_ASSIGNMENTS // experts // pad * pad + 1
    blocks = (experts - 1) * -(-per // pad)
    if per <= MAX_ASSIGNMENTS:
        assert sorted_row(blocks, pad, per - 1) == blocks * pad + per - 1


def test_the_kernels_use_it():
    """No other row arithmetic in the kernel that places the assignments."""
    text = open(os.path.join(mb_build.CSRC, "route_align.cu")).read()
    body = text[text.index("align_scatter_kernel("):]
    body = body[: body.index("\n}\n")]
    assert "sorted_row(" in body and "* pad" not in body
