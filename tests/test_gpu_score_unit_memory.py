"""Packed scores whose unit-gradient array cannot be allocated still give scores and gradients: the
backward then evaluates the Gaussians again.  Same scores bit for bit; gradients 1e-4 of the largest
component, as the two routes are compared elsewhere."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import autograd as ag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 200])
def test_no_memory_for_the_unit_gradient(cuda, monkeypatch, n):
    pts = torch.randn(4 * n, 4, device=cuda, generator=torch.Generator(cuda).manual_seed(n)) * 3
    off = torch.arange(5, dtype=torch.int32, device=cuda) * n
    one, idx = torch.zeros(4, dtype=torch.int32, device=cuda), torch.arange(4, device=cuda).int()
    leaf = pts.clone().requires_grad_()

    def run():
        s = ag.tanimoto_packed(pts[:n], off[:2], leaf, off, one, idx, lam=0.3)
        return s.detach(), torch.autograd.grad(s.sum(), leaf)[0]

    s, g = run()
    real, refused = torch.empty, []

    def empty(*shape, **kw):
        if shape == (4, n, 4):
            refused.append(shape)
            raise torch.OutOfMemoryError("CUDA out of memory")
        return real(*shape, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    s2, g2 = run()
    monkeypatch.undo()
    assert refused and torch.equal(s, s2)
    assert float((g - g2).abs().max()) < 1e-4 * float(g.abs().max())
