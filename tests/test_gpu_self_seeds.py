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
