"""The rule that gives a small cloud one block for its matrix and radius: its
points, each an odd number of floats apart, must fit the block's shared memory,
counted without wrapping (128 points of 2^25 coordinates are 2^32 floats). CPU
only."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("one") / "one.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(HERE, "dense_one_shim.cpp"),
                    "-o", so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("lp", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 64, 91, 92, 100, 127, 128, 129, 4096])
def test_rule(lib, n, lp):
    floats, points = lib.dense_one_floats(), lib.dense_one_points(lp)
    dims = {0, 1, 3, 64, 2**25, 2**26, 2**31, 2**32 - 1}
    for total in (floats, 2**32):   # both sides of the limit, and of the wrap
        dims |= {d for d in range(total // n - 3, total // n + 4) if 0 <= d < 2**32}
    for dim in dims:
        stride = lib.dense_one_stride(dim) & (2**32 - 1)
        assert stride % 2 == 1 and dim <= stride <= dim + 1
        assert bool(lib.dense_one_block(n, dim, lp)) == (n <= points and n * stride <= floats)
