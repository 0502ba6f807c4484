"""topo_loss over given bars, beside a plain loop over the clouds: uneven clouds,
clouds without bars, essential bars, and every kind of `top` (a negative one is
refused). The bars are made up, so no GPU is needed."""
import numpy as np
import pytest
import torch

from turbotops_gb300 import topo


def _bars(seed, counts):
    rng = np.random.default_rng(seed)
    h1 = np.concatenate([[0], np.cumsum(counts)])
    h0 = np.concatenate([[0], np.cumsum([c % 5 + 1 for c in counts])])
    t = lambda a: torch.from_numpy(np.asarray(a, np.float32)).requires_grad_()
    birth = rng.random(h1[-1])
    death = birth + rng.random(h1[-1])
    death[rng.random(h1[-1]) < 0.1] = np.inf
    return topo.Bars(t(rng.random(h0[-1])), t(birth), t(death), h0, h1, None, None, None)


def _plain(b, top):
    loss = 0.0
    for q in range(len(b.h0_offset) - 1):
        loss = loss + (b.h0_death[int(b.h0_offset[q]):int(b.h0_offset[q + 1])].double() ** 2).sum()
        s = slice(int(b.h1_offset[q]), int(b.h1_offset[q + 1]))
        p = (b.h1_death[s] - b.h1_birth[s])[torch.isfinite(b.h1_death[s])]
        if p.numel():
            loss = loss - torch.topk(p, min(top, p.numel())).values.double().sum()
    return loss


@pytest.mark.parametrize("top", [0, 1, 4, 1000])
@pytest.mark.parametrize("counts", [[7], [3, 0, 200, 1, 5], [0, 0], [40] * 30])
def test_loss_and_gradient(monkeypatch, counts, top):
    b = _bars(len(counts), counts)
    monkeypatch.setattr(topo, "diagrams", lambda *a, **k: b)
    got = topo.topo_loss(b.h0_death, [1], top=top)
    want = _plain(b, top)
    # FP32 sums of n terms: at most n 2^-24 of the terms' sizes
    n = b.h0_death.numel() + b.h1_birth.numel()
    size = float((b.h0_death ** 2).sum()) + b.h1_birth.numel()   # (every persistence is below 1)
    assert abs(got.item() - float(want)) <= n * 2.0**-24 * size
    for leaf in (b.h0_death, b.h1_birth, b.h1_death):
        g, h = (torch.autograd.grad(v, leaf, retain_graph=True, allow_unused=True)[0] for v in (got, want))
        zero = torch.zeros_like(leaf)
        assert torch.equal(zero if g is None else g, zero if h is None else h)


@pytest.mark.parametrize("top", [-1, -4, 0.5])
def test_refused_top(monkeypatch, top):
    b = _bars(3, [5, 9])
    monkeypatch.setattr(topo, "diagrams", lambda *a, **k: b)
    with pytest.raises((RuntimeError, TypeError)):
        topo.topo_loss(b.h0_death, [1], top=top)
