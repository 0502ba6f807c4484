"""The ranges of sorted edges that the spanning forest's rounds walk: for every
vertex and edge count they never fall and end at the last edge. CPU only."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def groups(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("groups") / "groups.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(HERE, "rank_groups_shim.cpp"),
                    "-o", so], check=True)
    L = C.CDLL(so)
    L.rank_groups.argtypes = [C.c_uint64, C.c_uint64, C.c_void_p]

    def f(m, n):
        e = (C.c_uint64 * 3)()
        L.rank_groups(m, n, e)
        return list(e)
    return f


def test_ends_never_fall(groups):
    ns = list(range(1, 200)) + [300, 1000, 1500, 1819, 1820, 1821, 2048, 2049, 4096, 8191, 8192, 8193, 16384, 16385,
                                100_000, 1_000_000, 2**31, 2**32 - 1]
    for n in ns:
        ms = {0, 1, 2**32 - 2}
        for at in (8 * n, 16 * n, 72 * n, 2**17, n * (n - 1) // 2):
            ms |= {at + k for k in (-1, 0, 1)}
        ms |= {int(2 ** (k / 4)) for k in range(128)}
        for m in sorted(ms):
            if not 0 <= m <= min(2**32 - 2, n * (n - 1) // 2):
                continue
            e = groups(m, n)
            assert e[0] <= e[1] <= e[2] == m, (m, n, e)
            if m < 16 * n or m < 2**17:
                assert e == [m, m, m]
            else:
                assert e[0] == 8 * n
