"""Dimension 1 by cocycles (dense_pairs_dim1) against the column reduction:
the same bars in the same order, critical simplices and pivots, on clouds with
one long class, many short ones, equal lengths (within a triangle and not),
duplicates, and at the sizes where a row's words begin. CPU only."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from turbotops_gb300 import synth

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "turbotops_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("cocycles") / "cocycles.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(HERE, "cocycle_shim.cpp"),
                    os.path.join(CSRC, "tt_reduce.cpp"), "-o", so, "-lpthread"], check=True)
    L = C.CDLL(so)
    P = C.c_void_p
    L.cocycles_agree.argtypes = [P, C.c_uint32, C.c_float, P, P, C.c_uint64, C.c_uint64, P]
    return L


def _agree(lib, x, metric="l2", thr=None, budget=1 << 32):
    mat = O.dense(x, metric)
    t = O.enclosing_radius(mat) if thr is None else np.float32(thr)
    r = O.dim0(mat=mat, thr=t, maxdim=1)
    mat = np.ascontiguousarray(mat, np.float32)
    ci, cd = np.ascontiguousarray(r["cidx"], np.uint64), np.ascontiguousarray(r["cd"], np.float32)
    bars = C.c_uint64()
    return lib.cocycles_agree(mat.ctypes.data, len(x), float(t), ci.ctypes.data, cd.ctypes.data, len(ci), budget,
                              C.byref(bars)), bars.value


@pytest.mark.parametrize("n", [2, 3, 4, 63, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("kind", ["circle", "gauss", "torus"])
def test_same_pairs(lib, kind, n):
    x = {"circle": lambda: synth.circles(1, n, seed=n)[0], "gauss": lambda: synth.gauss(n, 4, n),
         "torus": lambda: synth.torus(n, seed=n)}[kind]()
    for metric in ("l2", "l1", "linf"):
        assert _agree(lib, x, metric)[0] == 1


@pytest.mark.parametrize("seed", range(8))
def test_equal_lengths(lib, seed):
    """Rounded coordinates: groups of equal lengths, many within one triangle."""
    x = np.round(synth.gauss(40 + 25 * seed, 3, seed), 2 + seed % 2).astype(np.float32)
    x[-4:] = x[:4]   # duplicates: lengths of zero
    got, bars = _agree(lib, x)
    assert got == 1 and bars > 0


def test_batch_cloud_and_threshold(lib):
    x = synth.circle_batch(4, 300, 420)[2]
    assert _agree(lib, x)[0] == 1
    assert _agree(lib, x, thr=0.4)[0] == 1   # essential classes, several components


def test_declines(lib):
    assert _agree(lib, synth.lattice(200, dim=3, side=8))[0] == 2            # most lengths repeat
    assert _agree(lib, synth.circles(1, 200, seed=1)[0], budget=1000)[0] == 2
