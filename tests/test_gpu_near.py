"""The ordered searches (kNN lists and radius graphs over points in a spatial
order with box pruning) against the exhaustive scan of the same library and
the oracle, bit for bit: every padded dimension and lane order, tile and super
tile remainders, list lengths, ties, duplicates, outliers and non-finite
points."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, host
from oracle import oracle as O
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _cloud(kind, n, dim, seed):
    if kind == "grid":
        return synth.grid(n, dim, 50 if dim == 2 else 17, seed)
    if kind == "same":
        return np.full((n, dim), 0.25, np.float32)
    if kind == "gmm":
        return synth.gmm(n, dim, 5, seed)
    x = synth.gauss(n, dim, seed)
    if kind == "far":          # a common offset and a few outliers
        x += 3000.0
        x[:: max(1, n // 7)] *= 50.0
    elif kind == "nonfinite":  # NaN never enters a list, infinities sort last
        x[n // 3, 0] = np.nan
        x[n // 2, dim - 1] = np.inf
        x[n - 1] = -np.inf
        x[5] = np.nan
    return np.ascontiguousarray(x, np.float32)


def _lists(x, k, metric, mode):
    c = ctx()
    c.check(c.L.tt_ctx_set_knn_mode(c.h, mode))
    try:
        i, d = ops.knn(c, dev(x), k, metric)
        return host(i).view(np.uint32), bits(host(d))
    finally:
        c.check(c.L.tt_ctx_set_knn_mode(c.h, 0))


DIMS = (1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 24, 31, 33, 47, 48, 50, 63, 64)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("dim", DIMS + (32,))
def test_knn_every_dimension(dim, metric):
    x = _cloud("gmm" if dim > 8 else "gauss", 1100 + dim, dim, dim)
    for k in (1, 15):
        a, b = _lists(x, k, metric, 0), _lists(x, k, metric, 1)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert np.array_equal(a[0], O.knn(x, metric, 15))


@pytest.mark.parametrize("kind", ["grid", "same", "far", "nonfinite"])
@pytest.mark.parametrize("n,dim,k", [(512, 3, 32), (513, 2, 31), (1024, 3, 16), (1025, 4, 17), (2047, 2, 12),
                                     (1057, 8, 13), (4097, 3, 5)])
def test_knn_hard_clouds(kind, n, dim, k):
    x = _cloud(kind, n, dim, n)
    for metric in ("l2", "l1", "linf"):
        a, b = _lists(x, k, metric, 0), _lists(x, k, metric, 1)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("metric", ["lp:1.1", "lp:1.5", "lp:2.5", "lp:3", "lp:4", "lp:7.3", "lp:12", "lp:64"])
@pytest.mark.parametrize("kind,n,dim,k", [("gauss", 600, 2, 15), ("grid", 1025, 3, 16), ("gmm", 700, 8, 10),
                                          ("gauss", 640, 13, 7), ("gmm", 1500, 32, 15), ("gmm", 520, 50, 32),
                                          ("same", 530, 4, 5), ("far", 800, 5, 12), ("nonfinite", 700, 9, 8)])
def test_knn_lp(kind, n, dim, k, metric):
    """The Lp lists' power-sum filter and queue (exponents with and without a
    closed power, below and above 8 coordinates)."""
    x = _cloud(kind, n, dim, n)
    a, b = _lists(x, k, metric, 0), _lists(x, k, metric, 1)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e12, 1e25])
def test_knn_lp_scales(scale):
    """Powers that under- or overflow must filter nothing."""
    x = (synth.gauss(600, 10, 3) * np.float32(scale)).astype(np.float32)
    for metric in ("lp:1.5", "lp:3", "lp:9.5"):
        a, b = _lists(x, 12, metric, 0), _lists(x, 12, metric, 1)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
def test_knn_large_with_ties(metric):
    x = np.concatenate([synth.grid(20000, 3, 30, 4), synth.uniform(13000, 3, 5) * np.float32(30)])   # past 1,024 tiles
    a, b = _lists(x, 15, metric, 0), _lists(x, 15, metric, 1)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def _radius_check(x, tau, metric):
    rp, ci, w = ops.radius_graph(ctx(), dev(x), tau, metric)
    d = O.dense(x, metric)
    keep = d <= np.float32(tau)
    np.fill_diagonal(keep, False)
    r, c = np.nonzero(keep)
    assert np.array_equal(host(rp), np.concatenate([[0], np.cumsum(keep.sum(1))]))
    assert np.array_equal(host(ci), c.astype(np.int32))
    assert np.array_equal(bits(host(w)), bits(d[r, c]))


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("kind,n,dim,tau", [
    ("gauss", 600, 2, 0.05), ("gauss", 1500, 3, 0.6), ("gauss", 1025, 8, 2.5), ("grid", 900, 3, 2.0),
    ("grid", 900, 2, 3.0),                                  # boundary ties: d == tau is kept
    ("same", 700, 3, 0.0), ("same", 1025, 2, 0.5),          # rows of 699 and of 1,024: the longest ordered row
    ("same", 1026, 3, 0.5),                                 # 1,025: the exhaustive fill takes over
    ("gauss", 1300, 3, float("inf")), ("far", 800, 3, 1.0), ("gauss", 520, 12, 4.0)])
def test_radius(kind, n, dim, tau, metric):
    _radius_check(_cloud(kind, n, dim, n + dim), tau, metric)


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("kind,n,dim", [
    ("gauss", 512, 3), ("gauss", 1025, 2), ("gmm", 1100, 8), ("gmm", 2100, 12), ("gmm", 4200, 16), ("gmm", 1500, 32),
    ("gmm", 3000, 32), ("gmm", 1300, 50), ("gmm", 900, 64), ("grid", 2000, 3), ("grid", 1500, 2), ("same", 700, 3),
    ("far", 1200, 3), ("uniform", 33000, 3)])
def test_mst(kind, n, dim, metric):
    """Sorted spanning-tree weights: the ordered rounds against rounds that scan every pair."""
    x = dev(synth.uniform(n, dim, n) if kind == "uniform" else _cloud(kind, n, dim, n))
    c = ctx()
    a = bits(host(ops.mst_deaths(c, x, metric)))
    c.check(c.L.tt_ctx_set_knn_mode(c.h, 1))
    try:
        b = bits(host(ops.mst_deaths(c, x, metric)))
    finally:
        c.check(c.L.tt_ctx_set_knn_mode(c.h, 0))
    assert np.array_equal(a, b)


@pytest.mark.parametrize("order", ["random", "sorted", "striped"])
@pytest.mark.parametrize("n,tau", [(900, 0.9), (1400, 1.1), (2600, 1.0)])   # rows to 32, 512 and 1,024 entries
def test_radius_numbering(n, tau, order):
    """Row ids spread evenly, in one band (slots overflow), in stripes."""
    x = synth.gauss(n, 2, n)
    if order == "sorted":
        x = x[np.argsort(x[:, 0])]
    elif order == "striped":
        x = x[np.lexsort((x[:, 1], np.round(x[:, 0], 1)))]
    for t in (0.05, tau / 3, tau):
        _radius_check(np.ascontiguousarray(x), t, "l2")


def test_radius_wide_ids():
    """Rows whose ids spread over more than 2^22: sampled rows against all points."""
    n, tau = 4_400_000, np.float32(0.002)
    x = synth.uniform(n, 2, 3)
    rp, ci, w = (host(t) for t in ops.radius_graph(ctx(), dev(x), float(tau), "l2"))
    assert rp[0] == 0 and rp[-1] == len(ci)
    for i in (0, 1, 31, 32, 77777, n // 2, n - 1):
        a, b = int(rp[i]), int(rp[i + 1])
        d = x - x[i]
        dd = np.sqrt(d[:, 0].astype(np.float64) ** 2 + d[:, 1].astype(np.float64) ** 2)
        dd[i] = np.inf
        sure, maybe = np.flatnonzero(dd < tau * (1 - 1e-6)), np.flatnonzero(dd < tau * (1 + 1e-6))
        ids = ci[a:b]
        assert b - a > 20 and (np.diff(ids) > 0).all()
        assert set(sure) <= set(ids.tolist()) <= set(maybe.tolist())
        np.testing.assert_allclose(w[a:b], dd[ids], rtol=1e-6)
