"""Packed scores of a long reference against few fit points, whose overlap has a lane per reference
point, on both sides of a quarter of the warps' rows, for few pairs and for the many that take the
build with fewer registers: against a float64 evaluation, and the same score bits with and without
gradients.  Tolerances as in test_gpu_score_small: scores 1e-5, gradients 1e-4 of the largest
component."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import autograd as ag

pytestmark = pytest.mark.gpu


def _score64(x, y, lam):
    def v(a, b):
        e = -0.405 * ((a[:, None, :3] - b[None, :, :3]) ** 2).sum(-1)
        if lam:
            e = e - (a[:, None, 3] - b[None, :, 3]) ** 2 / lam
        return torch.exp(e).sum()
    ab = v(x, y)
    return ab / (v(x, x) + v(y, y) - ab)


@pytest.mark.parametrize("n,fits", [(512, [1, 2, 15, 16, 17, 31, 32, 33, 64]), (511, [3, 16, 0, 32]),
                                    (65, [1, 7, 8, 9, 16]), (64, [1, 15, 16, 17]), (300, [19, 20, 21])])
@pytest.mark.parametrize("lam", [None, 0.3])
@pytest.mark.parametrize("many", [False, True])
def test_few_fit_points(cuda, n, fits, lam, many):
    rng = np.random.default_rng(n)
    off = np.concatenate([[0], np.cumsum(fits)]).astype(np.int32)
    scale = [1, 1, 1, .1]
    P = 20 * torch.cuda.get_device_properties(cuda).multi_processor_count + 1 if many else len(fits)
    pf = np.arange(P, dtype=np.int32) % len(fits)
    g = lambda x, **k: torch.as_tensor(x, device=cuda, **k)
    ref = g(rng.uniform(-4, 4, (n, 4)) * scale, dtype=torch.float32)
    leaf = g(rng.uniform(-4, 4, (off[-1], 4)) * scale, dtype=torch.float32).requires_grad_()
    args = (ref, g(np.array([0, n], np.int32)), leaf, g(off), g(np.zeros(P, np.int32)), g(pf))
    s = ag.tanimoto_packed(*args, lam=lam)
    with torch.no_grad():
        assert torch.equal(s, ag.tanimoto_packed(*args, lam=lam))
    grad, = torch.autograd.grad(s.sum(), leaf)
    x, y = ref.double().cpu(), leaf.detach().double().cpu().requires_grad_()
    want = torch.stack([_score64(x, y[off[i]:off[i + 1]], lam) for i in range(len(fits))])
    used = torch.as_tensor(np.bincount(pf, minlength=len(fits)))
    g64, = torch.autograd.grad((want * used).sum(), y)
    np.testing.assert_allclose(s.detach().cpu().numpy(), want.detach().numpy()[pf], rtol=1e-5, atol=1e-9)
    d = grad.cpu().double() - g64
    assert float(d.abs().max()) < 1e-4 * float(g64.abs().max())
