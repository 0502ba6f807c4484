"""Matrix and radius of small clouds at the edges of the one-block kernel, bit
for bit against the oracle: the most points (128; 91 under Lp) and one more, odd
and even dimensions, the largest dimension that fits and the next."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, host
from oracle import oracle as O
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "l1", "linf", "lp:1.5", "lp:3"])
@pytest.mark.parametrize("n,dim", [(1, 1), (2, 64), (33, 32), (64, 16), (64, 187), (64, 188), (91, 3), (91, 131),
                                   (92, 3), (92, 32), (127, 2), (128, 31), (128, 32), (128, 93), (128, 94), (129, 8)])
def test_small_cloud(n, dim, metric):
    x = synth.gauss(n, dim, n + dim)
    mat, enc = ops.make_dense(ctx(), dev(x), metric)
    ref = O.dense(x, metric)
    assert np.array_equal(bits(host(mat)), bits(ref))
    assert bits(np.float32(enc)) == bits(O.enclosing_radius(ref))
