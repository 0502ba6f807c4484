"""Dimension 1 with the edges at hand (long columns swept, small complexes by
cocycles) against the plain column reduction: the same bars in the same order,
critical simplices, pivots and emergent counts, on clouds with one long class,
many short ones, equal lengths (within a triangle and not), duplicates,
thresholds, several threads, and where a row's words begin. CPU only."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from turbotops_gb300 import synth

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "turbotops_gb300", "csrc")
NEVER = 2**64 - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sweeps") / "sweeps.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", os.path.join(HERE, "sweep_shim.cpp"),
                    os.path.join(CSRC, "tt_reduce.cpp"), "-o", so, "-lpthread"], check=True)
    L = C.CDLL(so)
    P = C.c_void_p
    L.sweeps_agree.argtypes = [P, C.c_uint32, C.c_float, P, P, C.c_uint64, P, P, C.c_uint64, C.c_uint, P, P]
    return L


def _agree(lib, x, metric="l2", thr=None, patience=0, threads=1):
    """(agree, edges asked for, emergent pairs); patience 0: every column is swept."""
    mat = np.ascontiguousarray(O.dense(x, metric), np.float32)
    t = O.enclosing_radius(mat) if thr is None else np.float32(thr)
    r = O.dim0(mat=mat, thr=t, maxdim=1)
    ci, cd = np.ascontiguousarray(r["cidx"], np.uint64), np.ascontiguousarray(r["cd"], np.float32)
    e = O.emergent(mat=mat, cidx=ci, cd=cd)
    emi, emf = np.ascontiguousarray(e["emi"], np.uint64), np.ascontiguousarray(e["emf"], np.uint8)
    asked, emergent = C.c_uint32(), C.c_uint64()
    ok = lib.sweeps_agree(mat.ctypes.data, len(x), float(t), ci.ctypes.data, cd.ctypes.data, len(ci),
                          emi.ctypes.data, emf.ctypes.data, patience, threads, C.byref(asked), C.byref(emergent))
    return ok, asked.value, emergent.value


def _cloud(kind, n):
    if kind == "circle":
        return synth.circles(1, n, seed=n)[0]
    if kind == "torus":
        return synth.torus(n, seed=n)
    if kind == "eight":
        return synth.circle_batch(1, n, n, seed=n)[0]
    return synth.gauss(n, int(kind[5:]), n)


@pytest.mark.parametrize("n", [4, 63, 64, 65, 129, 255, 256, 257, 300, 320, 321, 385])
@pytest.mark.parametrize("kind", ["circle", "torus", "eight", "gauss3", "gauss16"])
def test_every_column_swept(lib, kind, n):
    x = _cloud(kind, n)
    for metric in ("l2", "l1", "linf") if n < 130 or n == 257 else ("l2",):
        assert _agree(lib, x, metric)[0] == 1


@pytest.mark.parametrize("threads", [1, 3])
@pytest.mark.parametrize("kind,n", [("circle", 512), ("torus", 700), ("eight", 400)])
def test_long_columns_are_swept(lib, kind, n, threads):
    ok, asked, _ = _agree(lib, _cloud(kind, n), patience=NEVER, threads=threads)
    assert ok == 1 and asked == 1
    assert _agree(lib, _cloud(kind, n), patience=0, threads=threads)[0] == 1


def test_short_columns_are_not(lib):
    for kind in ("gauss3", "gauss16"):
        assert _agree(lib, _cloud(kind, 300), patience=NEVER)[:2] == (1, 0)


@pytest.mark.parametrize("seed", range(10))
def test_equal_lengths(lib, seed):
    """Rounded coordinates: groups of equal lengths, many within one triangle,
    emergent pairs, duplicates (lengths of zero)."""
    n = 60 + 35 * seed   # on both sides of the cocycles' size
    x = np.round(synth.gauss(n, 3, seed), 2 + seed % 2).astype(np.float32)
    x[-4:] = x[:4]
    for patience in (0, 20_000, NEVER):
        assert _agree(lib, x, patience=patience)[0] == 1
    y = np.round(_cloud("circle", n), 2).astype(np.float32)
    assert _agree(lib, y)[0] == 1 and _agree(lib, y, "l1")[0] == 1


def test_emergent_pairs_are_counted_alike(lib):
    seen = 0
    for n, digits in ((120, 1), (200, 2), (256, 2), (300, 2), (420, 2)):
        ok, _, emergent = _agree(lib, np.round(synth.gauss(n, 3, n), digits).astype(np.float32))
        assert ok == 1
        seen += emergent
    assert seen > 0


def test_threshold_and_lattice(lib):
    x = _cloud("eight", 420)
    for t in (0.05, 0.2, 0.4, 1.0):   # essential classes, several components
        assert _agree(lib, x, thr=t)[0] == 1
    assert _agree(lib, synth.lattice(300, dim=3, side=8), "l1")[0] == 1   # most lengths repeat: the queue
