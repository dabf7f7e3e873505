"""Pharmacophore self overlaps (a warp per molecule, features by type) and start poses (four lanes
per pair) against the oracle at the sizes where their splits can go wrong: empty and one-feature
molecules, one feature more or less than a warp, several warps of features, ragged runs of pairs
that do not fill a warp, degenerate and non-finite clouds."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import kernels as K
from fast_shepherd_score_b200.layout import CloudSet, PharmSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directional,ext", [(True, 0), (True, 1), (True, 2), (False, 0)])
@pytest.mark.parametrize("copies", [1, 3000])
def test_pharm_self_overlap_sizes(cuda, directional, ext, copies):
    from oracle import align as oa
    rng = np.random.default_rng(8)
    sizes = [0, 1, 2, 8, 31, 32, 33, 63, 64, 65, 130]
    types = [rng.integers(0, 9, n) for n in sizes]
    anc = [(2.0 * rng.standard_normal((n, 3))).astype(np.float32) for n in sizes]
    vec = [rng.standard_normal((n, 3)).astype(np.float32) for n in sizes]
    rep = lambda a: [x for _ in range(copies) for x in a]
    ps = PharmSet.from_arrays(rep(types), rep(anc), rep(vec), device=cuda)
    got = K.pharm_self_overlap(ps, directional, ext).cpu().numpy().reshape(copies, len(sizes))
    pad = max(sizes)
    X, V = np.zeros((len(sizes), pad, 3), np.float32), np.zeros((len(sizes), pad, 3), np.float32)
    T = np.full((len(sizes), pad), 8, np.int32)
    for i, n in enumerate(sizes):
        X[i, :n], T[i, :n] = anc[i], types[i]
        V[i, :n] = vec[i] / np.linalg.norm(vec[i], axis=1, keepdims=True) if n else vec[i]
    want = oa.pharm_self_overlap(X, V, T, np.array(sizes), directionless=not directional, ext=ext)
    np.testing.assert_allclose(got, np.tile(want, (copies, 1)), rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("n_seeds", [1, 5, 6, 11, 12, 50, 64])
@pytest.mark.parametrize("pairs", [1, 7, 9, 33, 9500])
def test_seeds_sizes(cuda, n_seeds, pairs):
    from oracle import seeds as os_
    rng = np.random.default_rng(9)
    sizes = [1, 2, 3, 4, 5, 15, 16, 17, 33, 60, 129, 400]
    mk = lambda n: (rng.standard_normal((n, 3)) * np.array([5.0, 3.0, 2.0])).astype(np.float32)
    ref, fit = [mk(n) for n in sizes], [mk(n) for n in sizes]
    fit[8][5, 1] = np.nan     # non-finite: the fixed fallback set
    rs, fs = CloudSet.from_arrays(ref, device=cuda), CloudSet.from_arrays(fit, device=cuda)
    pr, pf = (np.arange(pairs) * 5) % len(sizes), (np.arange(pairs) * 7) % len(sizes)
    dev = lambda a: torch.from_numpy(a.astype(np.int32)).to(cuda)
    q, t = (x.cpu().numpy() for x in K.seeds(rs, fs, dev(pr), dev(pf), n_seeds))
    pad = max(sizes)
    P = lambda m: np.stack([np.pad(x, ((0, pad - len(x)), (0, 0))) for x in m])
    some = np.unique(np.concatenate([np.arange(min(pairs, 24)), [pairs - 1]]))
    N = np.array(sizes)
    wq, wt = os_.batched_seeds(P(ref)[pr[some]], P(fit)[pf[some]], N[pr[some]], N[pf[some]], n_seeds)
    ok = np.isfinite(wt).all((1, 2))
    # collinear and planar clouds (3 points or fewer) have no unique axes
    solid = ok & (N[pr[some]] > 3) & (N[pf[some]] > 3)
    np.testing.assert_allclose(q[some][solid], wq[solid], atol=2e-5)
    np.testing.assert_allclose(t[some][solid], wt[solid], atol=5e-5)
    np.testing.assert_allclose(np.linalg.norm(q[some], axis=-1), 1.0, atol=1e-5)
    few = (N[pr[some]] < 3) | (N[pf[some]] < 3)
    np.testing.assert_allclose(q[some][few], wq[few], atol=1e-6)
