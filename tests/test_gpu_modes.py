"""tt_ctx_set_knn_mode over radius graphs and spanning trees: modes 1 and 2 take
the exhaustive scans (fewer launches: no spatial order is made), and every mode
gives the same bits, at sizes past the CPU oracle's reach too."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, host
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _in_mode(mode, run):
    c = ctx()
    c.check(c.L.tt_ctx_set_knn_mode(c.h, mode))
    try:
        before = c.launches
        out = run(c)
        return out, c.launches - before
    finally:
        c.check(c.L.tt_ctx_set_knn_mode(c.h, 0))


@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("n,dim,tau", [(50_000, 3, 0.03), (2_000, 8, 1.0), (600, 1, 0.01)])
def test_radius(n, dim, tau, metric):
    x = dev(synth.uniform(n, dim, n))

    def run(c):
        rp, ci, w = ops.radius_graph(c, x, tau, metric)
        return host(rp), host(ci), bits(host(w))
    (a, la), (b, lb), (d, ld) = (_in_mode(m, run) for m in (0, 1, 2))
    for u, v, w in zip(a, b, d):
        assert np.array_equal(u, v) and np.array_equal(u, w)
    assert lb == ld and lb < la


@pytest.mark.parametrize("n,dim", [(3_000, 3), (20_000, 3), (2_000, 32), (600, 12)])
def test_mst(n, dim):
    x = dev(synth.uniform(n, dim, n))
    run = lambda c: bits(host(ops.mst_deaths(c, x, "l1" if dim == 12 else "l2")))
    (a, la), (b, lb), (d, ld) = (_in_mode(m, run) for m in (0, 1, 2))
    assert np.array_equal(a, b) and np.array_equal(a, d)
    assert lb < la
    assert ld == lb or dim == 32   # (in R^32 mode 2 takes the tensor-core lists)
