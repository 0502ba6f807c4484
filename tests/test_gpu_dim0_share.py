"""dim0 of dense complexes whose threshold keeps few or most of the pairs, on both
sides of the share from which the apparent scan goes by vertex pairs and of the
sizes that take one block (91) and no host round trip (1,280), bit for bit against
the oracle."""
import numpy as np
import pytest

from gpu_util import ctx, dev, host
from oracle import oracle as O
from test_gpu_dense_dim0 import _check_dim0, _check_emergent
from turbotops_gb300 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kept", [0, 1, "1/500", "1/16", "1/4-1", "1/4", "1/4+1", "1/2", "all"])
@pytest.mark.parametrize("kind,n", [("gauss", 2049), ("clusters", 2100), ("gauss", 3000), ("grid", 2100),
                                    ("gauss", 2), ("gauss", 91), ("gauss", 92), ("gauss", 1280), ("gauss", 1281),
                                    ("grid", 1281), ("grid", 92), ("grid", 91)])
def test_kept_share(kind, n, kept):
    x = {"gauss": lambda: synth.gauss(n, 3, n), "clusters": lambda: synth.gmm(n, 4, 7, n),
         "grid": lambda: synth.grid(n, 3, 17, n)}[kind]()
    mat, _ = ops.make_dense(ctx(), dev(x), "l2")
    m = host(mat)
    d = np.sort(m[np.tril_indices(n, -1)])
    pairs = len(d)
    count = {"1/500": pairs // 500, "1/16": pairs // 16, "1/4-1": -(-pairs // 4) - 1, "1/4": -(-pairs // 4),
             "1/4+1": pairs // 4 + 1, "1/2": pairs // 2, "all": pairs}.get(kept, kept)
    t = float(d[min(count, pairs) - 1]) if count else float(np.nextafter(d[0], np.float32(0)))
    r = ops.dim0(ctx(), mat=mat, threshold=t, maxdim=1)
    ref = O.dim0(mat=m, thr=t, maxdim=1)
    _check_dim0(r, ref)
    _check_emergent(r, O.emergent(mat=m, cidx=ref["cidx"], cd=ref["cd"]))
    assert int(host(r["tree"]).sum()) + r["essential"] == n
