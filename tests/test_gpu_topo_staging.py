"""The gradient step's clouds past its page-locked staging: clouds whose outputs
take more than its 256 MB give the bars they give one at a time."""
import numpy as np
import pytest
import torch

from gpu_util import bits, host
from turbotops_gb300 import synth, topo

pytestmark = pytest.mark.gpu


def test_more_than_the_staging_holds():
    n, count = 2048, 9   # 34 MB a cloud
    clouds = synth.circles(count, n, seed=9)
    x = torch.from_numpy(np.concatenate(clouds)).cuda()
    b = topo.diagrams(x, [n] * count)
    for q, y in enumerate(clouds):
        one = topo.diagrams(torch.from_numpy(y).cuda(), [n])
        s0, s1 = slice(*b.h0_offset[q:q + 2]), slice(*b.h1_offset[q:q + 2])
        assert np.array_equal(bits(host(b.h0_death[s0])), bits(host(one.h0_death)))
        assert np.array_equal(bits(host(b.h1_birth[s1])), bits(host(one.h1_birth)))
        assert np.array_equal(bits(host(b.h1_death[s1])), bits(host(one.h1_death)))
        assert np.array_equal(host(b.h1_death_edge[s1]) - q * n * (host(b.h1_death_edge[s1]) >= 0), host(one.h1_death_edge))
