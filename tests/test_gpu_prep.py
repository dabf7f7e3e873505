"""The launches around an alignment against plain float64 or integer forms: pair costs and index
flags, centred anchors, folded centroids, at sizes around a block and with empty molecules.
Tolerance 1e-6 of the coordinates' size: one subtraction, division or rotation in float32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 255, 256, 257, 5000])
def test_pair_cost_keys_and_range_flag(cuda, P):
    from fast_shepherd_score_b200 import kernels as K
    rng = np.random.default_rng(P)
    off = [np.concatenate([[0], np.cumsum(rng.integers(0, 70, 40))]).astype(np.int32)
           for _ in range(2)]
    pr, pf = (rng.integers(0, 40, P).astype(np.int32) for _ in range(2))
    t = [torch.as_tensor(x, device=cuda) for x in (*off, pr, pf)]
    key, bad = K.pair_cost(*t, 40, 40)
    assert (key.cpu().numpy() == -np.diff(off[0])[pr] * np.diff(off[1])[pf]).all()
    assert bad.item() == 0
    assert K.pair_cost(*t, 40, 40, check_range=False)[1] is None
    for k, v in ((2, -1), (3, 40), (2, 2 ** 31 - 1)):
        u = [x.clone() for x in t]
        u[k][P // 2] = v
        key, bad = K.pair_cost(*u, 40, 40)
        assert bad.item() == 1 and key[P // 2].item() == 0


@pytest.mark.parametrize("sizes", [[0], [1], [3, 0, 33, 70, 0], list(range(40))])
def test_centred_anchors(cuda, sizes):
    from fast_shepherd_score_b200 import kernels as K
    from fast_shepherd_score_b200.layout import PharmSet
    rng = np.random.default_rng(len(sizes))
    x = [rng.uniform(-20, 20, (n, 3)).astype(np.float32) for n in sizes]
    ty = [rng.integers(0, 9, n) for n in sizes]
    ph = PharmSet.from_arrays(ty, x, device=cuda)
    anc, pts, c = (v.cpu().numpy() for v in K.centre_anchors(ph))
    want = np.array([a.astype(np.float64).mean(0) if len(a) else np.zeros(3) for a in x])
    np.testing.assert_allclose(c, want, atol=2e-5)
    if sum(sizes):
        moved = np.concatenate([a - m for a, m in zip(x, c)])
        np.testing.assert_array_equal(anc[:, :3], moved)
        np.testing.assert_array_equal(pts[:, :3], moved)
        assert (anc[:, 3].view(np.int32) == np.concatenate(ty)).all() and not pts[:, 3].any()


@pytest.mark.parametrize("P", [1, 256, 300])
def test_folded_centroids(cuda, P):
    from fast_shepherd_score_b200 import align as al
    from fast_shepherd_score_b200 import kernels as K
    g = torch.Generator().manual_seed(P)
    q, t = torch.randn(P, 4, generator=g), torch.randn(P, 3, generator=g)
    cr, cf = 10 * torch.randn(7, 3, generator=g), 10 * torch.randn(5, 3, generator=g)
    pr, pf = torch.randint(0, 7, (P,), generator=g), torch.randint(0, 5, (P,), generator=g)
    got = K.fold_centroids(*(x.to(cuda) for x in (q, t, pr, pf, cr, cf))).cpu()
    R = al._quat_rot(q.double())
    want = t - torch.einsum("bij,bj->bi", R, cf.double()[pf]) + cr[pr]
    assert float((got - want).abs().max()) < 1e-6 * 60
