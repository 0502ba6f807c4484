"""dim0 of dense complexes at the edges of its kernels, bit for bit against the
oracle: the apparent scan's lanes (32 edges of a row) and candidate limits
(64 per lane, then the whole warp; 32 for the emergent probe), and the
spanning forest's rank groups (8 n and 72 n edges)."""
import numpy as np
import pytest

from gpu_util import bits, ctx, dev, h0_pairs, host
from oracle import oracle as O
from test_gpu_dense_dim0 import _check_dim0, _check_emergent
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


def _clumps(n, seed):
    """Tight pairs far apart, then outliers: short edges without any cofacet,
    and cofacets that only low vertex numbers offer."""
    rng = np.random.default_rng(seed)
    base = rng.normal(0, 10, ((n + 1) // 2, 3))
    x = np.concatenate([base, base + rng.normal(0, 1e-3, base.shape)])[:n]
    x[-3:] += 1000.0 * np.arange(1, 4)[:, None]
    return np.ascontiguousarray(x, np.float32)


CASES = [("gauss", n, "inf") for n in (2, 3, 31, 32, 33, 64, 65, 72, 73, 129)]
CASES += [("clumps", n, t) for n in (33, 97, 200, 400) for t in ("inf", "2.5")]
CASES += [("grid", n, "inf") for n in (34, 100, 300)]        # ties: emergent probes past 32 candidates
CASES += [("gauss", 2048, "inf"), ("clumps", 2048, "60"), ("gauss", 2049, "inf"), ("clumps", 2100, "60")]   # one block's forest, separate rounds
CASES += [("same", 70, "inf"), ("gauss", 700, "0.35"), ("clumps", 700, "30")]   # m below and above 16 n


@pytest.mark.parametrize("kind,n,thr", CASES)
def test_dim0_pairs(kind, n, thr):
    if kind == "clumps":
        x = _clumps(n, n)
    elif kind == "same":
        x = np.zeros((n, 3), np.float32)
    else:
        x = synth.grid(n, 2, 24, n) if kind == "grid" else synth.gauss(n, 3, n)
    mat, enc = ops.make_dense(ctx(), dev(x), "l1" if kind == "grid" else "l2")
    t = enc if thr == "inf" else float(np.float32(thr))
    r = ops.dim0(ctx(), mat=mat, threshold=t, maxdim=1)
    m = host(mat)
    ref = O.dim0(mat=m, thr=t, maxdim=1)
    _check_dim0(r, ref)
    _check_emergent(r, O.emergent(mat=m, cidx=ref["cidx"], cd=ref["cd"]))
    assert int(host(r["tree"]).sum()) + r["essential"] == n
    r0 = ops.dim0(ctx(), mat=mat, threshold=t, maxdim=0)
    assert np.array_equal(bits(h0_pairs(r0)), bits(ref["h0"])) and np.array_equal(host(r0["keys"]), host(r["keys"]))
