"""The ordered lists above 8 coordinates where their kernels change: the table of
separations from 2,048 points on, half as many queries a warp up to 10,000, and
the full number beyond, against the exhaustive scan, bit for bit, on clusters
(blocks are left out), one Gaussian (hardly any), a far offset with outliers,
duplicates and non-finite points."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_near import _cloud, _lists
from turbotops_gb300 import synth

pytestmark = pytest.mark.gpu


def _make(kind, n, dim):
    if kind == "twins":   # every point four times: ties across tiles
        return np.ascontiguousarray(np.tile(synth.gauss((n + 3) // 4, dim, n), (4, 1))[:n])
    return _cloud(kind, n, dim, n + dim)


def _same(x, k, metric):
    a, b = _lists(x, k, metric, 0), _lists(x, k, metric, 1)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    return a


SIZES = (2047, 2048, 2049, 10_000, 10_001, 12_003)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("dim", [9, 16, 17, 24, 33, 48, 64])
@pytest.mark.parametrize("n", SIZES)
def test_lists(n, dim, metric):
    for kind, k in (("gmm", 15), ("gauss", 7)):
        _same(_make(kind, n, dim), k, metric)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf", "lp:1.5", "lp:3", "lp:2.5"])
@pytest.mark.parametrize("kind", ["far", "nonfinite", "twins"])
@pytest.mark.parametrize("n,dim,k", [(2049, 24, 32), (10_001, 12, 15), (10_500, 33, 17), (11_000, 64, 5)])
def test_hard_clouds(n, dim, k, kind, metric):
    _same(_make(kind, n, dim), k, metric)


@pytest.mark.parametrize("metric", ["lp:1.5", "lp:3", "lp:2.5", "lp:1", "lp:20"])
@pytest.mark.parametrize("n,dim", [(2048, 16), (2049, 32), (10_000, 9), (10_001, 9), (10_001, 24), (12_003, 48),
                                   (12_003, 64)])
def test_lp(n, dim, metric):
    for kind, k in (("gmm", 15), ("gauss", 6)):
        _same(_make(kind, n, dim), k, metric)


@pytest.mark.parametrize("metric", ["l1", "lp:3"])
def test_against_the_oracle(metric):
    x = _make("gmm", 10_001, 24)
    a = _same(x, 12, metric)
    rows = O.knn_rows(x, metric, 12, 0, len(x), 16)
    assert np.array_equal(a[0], rows)
