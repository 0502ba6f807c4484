"""A buffer that only grows: after an allocation that failed it holds nothing and
claims nothing, and the next request allocates. CPU only."""
import ctypes as C
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_growth(tmp_path):
    so = str(tmp_path / "grow.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(HERE, "grow_shim.cpp"), "-o", so],
                   check=True)
    L = C.CDLL(so)

    def grow(want, fail=0):
        b, h = C.c_uint64(), C.c_int()
        return L.grow(C.c_uint64(want), fail, C.byref(b), C.byref(h)), b.value, h.value
    assert grow(100) == (0, 100, 1)
    assert grow(50, 1) == (0, 100, 1)      # large enough: nothing to allocate
    assert grow(200, 1) == (1, 0, 0)       # failed: empty, the old memory given back
    assert grow(100) == (0, 100, 1)        # (a stale size would hand out no memory)
    assert grow(300) == (0, 300, 1)
