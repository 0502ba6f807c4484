"""Long columns of whole calls: a circle in a Gaussian cloud of R^32 has more than
4,096 columns (several reducing threads) and one long one, for which a reducing
thread asks for the edges in order. The bars are those of the gradient step's
reduction, which has the edges at hand and one thread."""
import numpy as np
import pytest
import torch

from gpu_util import bits, host
from turbotops_gb300 import api, synth, topo

pytestmark = pytest.mark.gpu


def _cloud(n, m, seed):
    rng = np.random.default_rng(seed)
    t = rng.uniform(0, 2 * np.pi, m)
    c = rng.normal(0, 0.1, (m, 32))
    c[:, 0] += 6 * np.cos(t)
    c[:, 1] += 6 * np.sin(t)
    return np.concatenate([synth.gauss(n, 32, seed), c.astype(np.float32)])


@pytest.mark.parametrize("x", [_cloud(1900, 500, 1), synth.circles(1, 700, seed=2)[0], synth.torus(800, seed=3),
                               synth.circles(1, 256, seed=4)[0], synth.circles(1, 257, seed=5)[0]],
                         ids=["threads", "circle", "torus", "256", "257"])
def test_same_bars(x):
    dgms, info = api.persistence(x, maxdim=1)
    if len(x) == 2400:
        assert info["columns"][0] > 4096
    b = topo.diagrams(torch.from_numpy(x).cuda(), [len(x)], threads=1)
    assert np.array_equal(bits(dgms[1][:, 0]), bits(host(b.h1_birth)))
    assert np.array_equal(bits(dgms[1][:, 1]), bits(host(b.h1_death)))
