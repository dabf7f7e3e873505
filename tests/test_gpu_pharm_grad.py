"""Mode "pharm": the translations carry the centroids' share of the anchors' gradient, backwards and
forwards.  t = t' - R c_fit + c_ref with c the mean of a molecule's anchors, so w . t pulls
w / n on every reference anchor and -R^T w / n on every fit anchor.  Tolerance 1e-5: sums of at most
three float32 products of size one, divided by up to 9."""
import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200 import api
from fast_shepherd_score_b200.layout import PharmSet

pytestmark = pytest.mark.gpu


def _sets(cuda, sizes=(4, 9, 0, 1)):
    rng = np.random.default_rng(3)
    mk = lambda: PharmSet.from_arrays([rng.integers(0, 8, n) for n in sizes],
                                      [rng.uniform(-5, 5, (n, 3)) for n in sizes],
                                      [rng.standard_normal((n, 3)) for n in sizes], device=cuda)
    idx = torch.arange(len(sizes), dtype=torch.int32, device=cuda)
    return mk(), mk(), idx, np.array(sizes)


def _run(r, f, idx):
    return api.align_device("pharm", None, None, r, f, idx, idx, num_seeds=8, steps=5)


@pytest.mark.parametrize("side", ["ref", "fit", "both"])
def test_translation_gradient(cuda, side):
    r, f, idx, n = _sets(cuda)
    plain = _run(r, f, idx)
    assert not plain[2].requires_grad
    r.anc.requires_grad_(side != "fit")
    f.anc.requires_grad_(side != "ref")
    with torch.no_grad():
        assert not _run(r, f, idx)[2].requires_grad
    sc, q, t = _run(r, f, idx)
    torch.testing.assert_close(t.detach(), plain[2], atol=1e-5, rtol=0)
    assert torch.equal(sc, plain[0]) and torch.equal(q, plain[1])
    w = torch.randn(t.shape, device=cuda, generator=torch.Generator(cuda).manual_seed(1))
    leaves = [x.anc for x in (r, f) if x.anc.requires_grad]
    got = list(torch.autograd.grad((w * t).sum(), leaves))
    mol = torch.as_tensor(np.repeat(np.arange(len(n)), n), device=cuda)
    share = 1.0 / torch.as_tensor(n, device=cuda).clamp(min=1)[:, None]
    for s, g in (("ref", w), ("fit", -torch.einsum("bij,bi->bj", al._quat_rot(q), w))):
        if side in (s, "both"):
            d = got.pop(0)
            torch.testing.assert_close(d[:, :3], (g * share)[mol], atol=1e-5, rtol=0)
            assert not d[:, 3].any()


def test_translation_tangent(cuda):
    r, f, idx, n = _sets(cuda)
    v = torch.ones_like(r.anc)
    with forward_ad.dual_level():
        r.anc = forward_ad.make_dual(r.anc, v)
        tan = forward_ad.unpack_dual(_run(r, f, idx)[2]).tangent
    want = torch.as_tensor(n > 0, device=cuda).float()[:, None].expand(-1, 3)
    torch.testing.assert_close(tan, want, atol=1e-5, rtol=0)
