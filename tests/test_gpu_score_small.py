"""GPU parity of the packed scores of clouds of up to 512 points and their gradients with a float64 evaluation,
at the sizes where a cloud changes its rows per lane or its padding, with a shared reference, with
changing ones and with molecules of several pairs.  Tolerances: scores 1e-5 (float32 sums of
Gaussians), gradients 1e-4 relative to the largest component, as test_gpu_kernels has them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64]
WIDE = [65, 100, 127, 128, 129, 200, 256, 257, 400, 511, 512]


def _set(rng, sizes, spread):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    pts = rng.uniform(-spread, spread, (int(off[-1]), 4))
    pts[:, 3] = rng.uniform(-.3, .3, len(pts))
    return pts.astype(np.float32), off


def _score64(x, y, lam):
    def v(a, b):
        e = -0.405 * ((a[:, None, :3] - b[None, :, :3]) ** 2).sum(-1)
        if lam is not None:
            e = e - (a[:, None, 3] - b[None, :, 3]) ** 2 / lam
        return torch.exp(e).sum()
    ab = v(x, y)
    return ab / (v(x, x) + v(y, y) - ab)


@pytest.mark.parametrize("lam", [None, 0.3])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("sizes,repeat", [(SIZES, 1), (SIZES, 400), (WIDE + [1, 64], 1)])
def test_small_scores_and_gradients(cuda, lam, shared, sizes, repeat):
    from fast_shepherd_score_b200 import autograd as ag
    rng = np.random.default_rng(5)
    rp, ro = _set(rng, sizes, 3.)
    fp, fo = _set(rng, sizes[::-1], 3.)
    n = len(sizes)
    pf = np.tile(np.arange(n, dtype=np.int32), repeat)
    pr = np.full_like(pf, 9) if shared else ((pf * 4 + 1) % n).astype(np.int32)
    t = {k: torch.as_tensor(v, device=cuda) for k, v in
         dict(rp=rp, ro=ro, fp=fp, fo=fo, pr=pr, pf=pf).items()}
    leaf = t["fp"].clone().requires_grad_()
    w = torch.linspace(0.5, 1.5, len(pf), device=cuda)
    got = ag.tanimoto_packed(t["rp"], t["ro"], leaf, t["fo"], t["pr"], t["pf"], lam=lam)
    grad, = torch.autograd.grad((got * w).sum(), leaf)
    with torch.no_grad():
        plain = ag.tanimoto_packed(t["rp"], t["ro"], leaf, t["fo"], t["pr"], t["pf"], lam=lam)
    assert torch.equal(plain, got)
    # both sides differentiated: the other route of the backward
    both = t["rp"].clone().requires_grad_()
    two = ag.tanimoto_packed(both, t["ro"], leaf, t["fo"], t["pr"], t["pf"], lam=lam)
    assert torch.equal(two, got)
    other = torch.autograd.grad((two * w).sum(), (leaf, both))[0]

    x64 = torch.as_tensor(rp, dtype=torch.float64)
    y64 = torch.as_tensor(fp, dtype=torch.float64).requires_grad_()
    wf = np.zeros(n)
    np.add.at(wf, pf, w.cpu().numpy().astype(np.float64))
    ref = torch.stack([_score64(x64[ro[pr[i]]:ro[pr[i] + 1]], y64[fo[i]:fo[i + 1]], lam)
                       for i in range(n)])
    g64, = torch.autograd.grad((ref * torch.as_tensor(wf)).sum(), y64)
    np.testing.assert_allclose(got.detach().cpu().numpy(), np.tile(ref.detach().numpy(), repeat),
                               rtol=1e-5)
    scale = float(g64.abs().max())
    for g in (grad, other):
        assert float((g.cpu().double() - g64).abs().max()) < 1e-4 * scale
    if lam is None:
        assert not grad[:, 3].any()


def test_small_scores_of_bad_pairs_and_empty_clouds(cuda):
    from fast_shepherd_score_b200 import autograd as ag
    rng = np.random.default_rng(6)
    rp, ro = _set(rng, [20, 0, 30], 3.)
    fp, fo = _set(rng, [10, 0, 40, 12], 3.)
    t = [torch.as_tensor(v, device=cuda) for v in (rp, ro, fp, fo)]
    pr = torch.tensor([0, 0, 0, 1, 2, 0], dtype=torch.int32, device=cuda)
    pf = torch.tensor([0, 1, 2, 3, 3, 3], dtype=torch.int32, device=cuda)
    leaf = t[2].clone().requires_grad_()
    # pairs 2 and 4 exceed the declared sizes: NaN and no gradient
    s = ag.tanimoto_packed(t[0], t[1], leaf, t[3], pr, pf, max_ref=20, max_fit=30)
    g, = torch.autograd.grad(s[[0, 1, 3, 5]].sum(), leaf)
    s = s.detach().cpu()
    assert torch.isnan(s[[2, 4]]).all() and torch.isfinite(s[[0, 1, 3, 5]]).all()
    assert float(s[1]) == 0.0 and float(s[3]) == 0.0
    assert torch.isfinite(g).all() and not g[10:50].any() and g[50:].any()
