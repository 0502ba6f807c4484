"""The spanning forest of graph complexes at the edges of its rank groups (16 n,
72 n and 2^17 edges): dim0 of a caller's CSR and of a radius graph, and
persistence with a threshold, bit for bit against the oracle, on clouds that
end in one component and in several."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, h0_pairs, host
from oracle import oracle as O
from test_gpu_dense_dim0 import _check_dim0
from turbotops_gb300 import api, ops, synth

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    if kind == "torus":
        return synth.torus(n, seed=n)
    x = synth.uniform(n, 3, n)
    if kind == "parts":   # four parts that no threshold here joins, and two single points
        x[:, 0] += 100.0 * (np.arange(n) % 4)
        x[-2:] += np.float32([[0, 500, 0], [0, 900, 0]])
    return x


def _threshold(x, m):
    """The m-th smallest pair length: a graph of m edges (more where it ties)."""
    d = O.dense(x, "l2")[np.tril_indices(len(x), -1)]
    return float(np.partition(d, m - 1)[m - 1])


CASES = [("torus", 1000, 120_408), ("uniform", 300, 26_910), ("uniform", 1000, 99_900), ("uniform", 1500, 123_667)]
for _n in (300, 1000, 1500, 1819, 1821):
    for _m in (16 * _n - 1, 16 * _n, 72 * _n - 1, 72 * _n + 1, 2**17 - 1, 2**17, 2**17 + 1):
        if _m < _n * (_n - 1) // 2:
            CASES.append(("uniform", _n, _m))
for _n, _ms in ((300, (4_900, 10_800)), (1000, (16_100, 72_001, 99_000)), (1500, (23_999, 108_001, 131_000)),
                (1819, (130_969, 131_071, 131_072)), (2500, (2**17 - 1, 2**17, 180_001))):
    CASES += [("parts", _n, _m) for _m in _ms]


@pytest.mark.parametrize("kind,n,m", CASES)
def test_graph_forest(kind, n, m):
    x = _cloud(kind, n)
    t = _threshold(x, m)
    rp, ci, w = O.radius_graph(x, "l2", np.float32(t))
    assert len(ci) // 2 >= m
    ref = O.dim0(csr=(rp, ci, w), n=n, thr=t, maxdim=1)
    csr = (dev(rp.view(np.int64)), dev(ci.view(np.int32)), dev(w))
    r = ops.dim0(ctx(), csr=csr, n=n, threshold=t, maxdim=1)
    _check_dim0(r, ref)
    assert int(host(r["tree"]).sum()) + r["essential"] == n
    assert (r["essential"] > 1) or kind != "parts"
    g = ops.radius_graph(ctx(), dev(x), t, "l2")
    r0 = ops.dim0(ctx(), csr=g, n=n, threshold=t, maxdim=0)
    assert np.array_equal(bits(h0_pairs(r0)), bits(ref["h0"])) and np.array_equal(host(r0["keys"]), host(r["keys"]))


@pytest.mark.parametrize("kind,n,m", [("torus", 1000, 120_408), ("uniform", 1000, 99_900), ("parts", 300, 10_000),
                                      ("parts", 1500, 123_667)])
def test_persistence_with_threshold(kind, n, m):
    x = _cloud(kind, n)
    t = float(np.float32(_threshold(x, m)))
    rp, ci, w = O.radius_graph(x, "l2", np.float32(t))
    ref = O.dim0(csr=(rp, ci, w), n=n, thr=t, maxdim=1)["h0"]
    a, _ = api.persistence(x, maxdim=1, threshold=t)
    assert np.array_equal(bits(a[0].ravel()), bits(ref))
    b, _ = api.persistence_graph(rp, ci, w, n, maxdim=1, threshold=t)
    assert np.array_equal(api.canonical(a), api.canonical(b))
