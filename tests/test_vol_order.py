"""The volumetric kernels deal their work items out over the warps: every item
is taken exactly once, whatever the remainders, and the numbers one warp takes
together lie far apart. CPU only."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "vol_order_host.cu")


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("vol_order") / "libvolorder.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC",
                    "-ccbin", "/usr/bin/g++", "-o", out, SRC], check=True)
    lib = C.CDLL(out)

    def order(total, lanes, warps):
        a = np.zeros(max(total, 1), dtype=np.uint32)
        lib.vol_deal(C.c_uint(total), C.c_uint(lanes), C.c_uint(warps), a.ctypes.data_as(C.c_void_p))
        return a[:total].astype(np.int64)

    return order


@pytest.mark.parametrize("lanes,warps", [(1, 1), (1, 4), (3, 4), (32, 1), (32, 8), (5, 1776), (32, 1776)])
def test_dealing_order_is_a_permutation(deal, lanes, warps):
    block = lanes * warps
    for total in sorted({1, 2, lanes, max(block - 1, 1), block, block + 1, 2 * block - 1, 2 * block}):
        got = deal(total, lanes, warps)
        assert np.array_equal(np.sort(got), np.arange(total)), total
        # a warp's first takes: one from each row of the (last) block
        m = min(total, block)
        first = got[:min(lanes, m)]
        if m >= lanes:
            assert np.all(np.diff(first) >= m // lanes)
