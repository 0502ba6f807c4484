"""The batch where its distances crowd or its clouds are large, against the
per-cloud entry points bit for bit: slots of an item with ties (ordered by a
warp, up to 512) and with distances that only nearly tie, clouds on both sides
of the size that has no items, and the radix passes over clouds with and
without a block for every tile."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, host
from test_gpu_batch_bins import _line, _tight
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _rings(n, copies):   # every distance of a regular polygon `copies` times and more
    t = 2 * np.pi * (np.arange(n) % (n // copies)) / (n // copies)
    return np.c_[np.cos(t), np.sin(t), np.zeros(n)].astype(np.float32)


GROUPS = {
    "ties": lambda: [synth.lattice(n, n, s, 3) for n, s in ((120, 6), (300, 20), (500, 9), (1000, 20))]
    + [_line(n) for n in (64, 130, 258, 300, 514, 520, 700)] + [_rings(240, 4), _rings(600, 3)],
    "near_ties": lambda: [_tight(n, n) for n in (12, 20, 32, 40, 45, 46, 60, 64)],
    "both": lambda: [np.concatenate([synth.lattice(200, 1, 8, 3), _tight(40, 2)]), synth.gauss(900, 3, 4)],
    "sizes": lambda: [synth.gauss(5017, 3, 1), synth.uniform(90, 3, 2), synth.gauss(5018, 3, 3), synth.uniform(4400, 3, 4)],
    "large_only": lambda: [synth.gauss(5018, 3, 5)],
    "tied_large": lambda: [synth.lattice(3000, i, 20, 3) for i in range(4)],
    "one_point": lambda: [synth.gauss(1, 3, 1)] * 3,
}


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("group", list(GROUPS))
def test_batch(group, metric, use_graph):
    clouds = GROUPS[group]()
    b = ops.DenseBatch(ctx(), [c.shape[0] for c in clouds], 3, metric, use_graph=use_graph)
    b.load(dev(np.concatenate(clouds)))
    for _ in range(2):
        b.run()
    r = b.result()
    off, d_all, v_all = host(r["edge_offset"]), host(r["diam"]), host(r["verts"])
    for q, x in enumerate(clouds):
        mat, enc = ops.make_dense(ctx(), dev(x), metric)
        assert bits(host(r["radius"])[q]) == bits(np.float32(enc)), q
        d, v = ops.redzed_edges(ctx(), mat=mat, threshold=enc)
        s, e = int(off[q]), int(off[q + 1])
        assert np.array_equal(bits(d_all[s:e]), bits(host(d))), q
        assert np.array_equal(v_all[2 * s:2 * e], host(v)), q
    b.close()
