"""Packed scores of small clouds on both sides of the pair counts where a pair changes from a warp for
16 rows to 32 and to one warp, against a float64 evaluation.  Tolerances as in test_gpu_score_small:
scores 1e-5, gradients 1e-4 of the largest component."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import autograd as ag

pytestmark = pytest.mark.gpu


def _score64(x, y, lam):
    def v(a, b):
        e = -0.405 * ((a[:, None, :3] - b[None, :, :3]) ** 2).sum(-1)
        return torch.exp(e - (a[:, None, 3] - b[None, :, 3]) ** 2 / lam).sum()
    ab = v(x, y)
    return ab / (v(x, x) + v(y, y) - ab)


@pytest.mark.parametrize("sizes", [[1, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64], [1, 2, 7, 16], [33]])
@pytest.mark.parametrize("per_sm,more", [(0, 1), (3, 0), (3, 1), (6, 0), (6, 1)])
def test_scores_by_number_of_pairs(cuda, sizes, per_sm, more):
    P = per_sm * torch.cuda.get_device_properties(cuda).multi_processor_count + more
    rng = np.random.default_rng(len(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    pts = [rng.uniform(-3, 3, (off[-1], 4)).astype(np.float32) * [1, 1, 1, .1] for _ in range(2)]
    n = len(sizes)
    pf = np.arange(P, dtype=np.int32) % n
    pr = (pf * 3 + 1) % n
    g = lambda x, **k: torch.as_tensor(x, device=cuda, **k)
    ref, leaf = (g(p, dtype=torch.float32) for p in pts)
    leaf.requires_grad_()
    s = ag.tanimoto_packed(ref, g(off), leaf, g(off), g(pr), g(pf), lam=0.3)
    grad, = torch.autograd.grad(s.sum(), leaf)
    x, y = (t.detach().double().cpu() for t in (ref, leaf))
    y.requires_grad_()
    used = np.bincount(pf, minlength=n)
    want = torch.stack([_score64(x[off[(i * 3 + 1) % n]:off[(i * 3 + 1) % n + 1]],
                                 y[off[i]:off[i + 1]], 0.3) for i in range(n)])
    g64, = torch.autograd.grad((want * torch.as_tensor(used)).sum(), y)
    np.testing.assert_allclose(s.detach().cpu().numpy(), want.detach().numpy()[pf], rtol=1e-5)
    assert float((grad.cpu().double() - g64).abs().max()) < 1e-4 * float(g64.abs().max())
