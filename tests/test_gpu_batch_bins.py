"""The batch's bin partition at its limits, against the per-cloud entry points
bit for bit: clouds of 1 and 2 points, bins that overflow (ties, duplicates,
tight clusters) beside clouds that do not, item and chunk remainders, crowded
items."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, host
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _line(n):      # distances of one value each, evenly spread
    x = np.zeros((n, 3), np.float32)
    x[:, 0] = np.arange(n)
    return x


def _tight(n, seed):   # two far clusters: almost every distance in two narrow bands
    x = np.random.default_rng(seed).normal(0, 1e-4, (n, 3))
    x[n // 2:, 0] += 5.0
    return x.astype(np.float32)


GROUPS = {
    "mixed": lambda: [synth.uniform(1, 3, 1), synth.uniform(2, 3, 2), synth.grid(700, 3, 9, 3), synth.uniform(300, 3, 4),
                      np.zeros((600, 3), np.float32), synth.gauss(1024, 3, 5), _tight(900, 6), _line(400),
                      synth.uniform(65, 3, 7)],
    "no_radix": lambda: [synth.uniform(n, 3, n) for n in (3, 64, 91, 129, 512, 513, 1500, 2049)],
    "all_radix": lambda: [np.ones((500, 3), np.float32), synth.grid(1000, 3, 10, 1), synth.grid(729, 3, 9, 2)],
    "crowded_items": lambda: [synth.grid(60, 3, 8, 3), _line(200), np.full((40, 3), 2, np.float32)],
    "one_large": lambda: [synth.gauss(5000, 3, 9)],   # many chunks of one cloud
}


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("metric", ["l2", "l1", "linf"])
@pytest.mark.parametrize("group", list(GROUPS))
def test_batch_bins(group, metric, use_graph):
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


def test_batch_bins_follow_the_points():
    """The same batch on other points: no count of an earlier run survives."""
    a, c = synth.uniform(800, 3, 1), synth.grid(800, 3, 10, 2)
    b = ops.DenseBatch(ctx(), [800, 800], 3, "l2")
    for first, second in ((a, c), (c, a), (a, a), (c, c)):
        b.load(dev(np.concatenate([first, second])))
        b.run()
        r = b.result()
        off = host(r["edge_offset"])
        for q, x in enumerate((first, second)):
            mat, enc = ops.make_dense(ctx(), dev(x), "l2")
            d, v = ops.redzed_edges(ctx(), mat=mat, threshold=enc)
            s, e = int(off[q]), int(off[q + 1])
            assert np.array_equal(bits(host(r["diam"])[s:e]), bits(host(d)))
            assert np.array_equal(host(r["verts"])[2 * s:2 * e], host(v))
    b.close()
