"""GPU parity of the padded pose evaluations with the float64 oracle at the sizes where a pose
changes its warps, its lanes or its register tile, with padding and without, and with poses left
over in the last warp.  Tolerances as in test_gpu_kernels: values 1e-5, gradients 1e-4 relative to
the row's largest component; where the terms cancel, relative to the pose's overlap, which is the
size of the terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _poses(K, N, M, seed, ragged):
    rng = np.random.default_rng(seed)
    q = rng.standard_normal((K, 4))
    d = {"A": rng.uniform(-4, 4, (K, N, 3)), "B": rng.uniform(-4, 4, (K, M, 3)),
         "RV": rng.standard_normal((K, N, 3)), "FV": rng.standard_normal((K, M, 3)),
         "CA": rng.uniform(-.3, .3, (K, N)), "CB": rng.uniform(-.3, .3, (K, M)),
         "q": q / np.linalg.norm(q, axis=1, keepdims=True), "t": rng.uniform(-1, 1, (K, 3))}
    d = {k: v.astype(np.float32) for k, v in d.items()}
    d.update(At=rng.integers(0, 9, (K, N)).astype(np.int32),
             Bt=rng.integers(0, 9, (K, M)).astype(np.int32), Nr=None, Mr=None)
    if ragged:
        d.update(Nr=rng.integers(0, N + 1, K).astype(np.int32),
                 Mr=rng.integers(0, M + 1, K).astype(np.int32))
    return d


def _check(got, ref, need_grad):
    V, dQ, dT = (x.cpu().numpy() for x in got)
    np.testing.assert_allclose(V, ref[0], rtol=1e-5, atol=1e-6)
    for g, r in ((dQ, ref[1]), (dT, ref[2])):
        if need_grad:
            scale = np.abs(r).max(1, keepdims=True) + np.abs(ref[0])[:, None] + 1e-2
            assert np.max(np.abs(g - r) / scale) < 1e-4
        else:
            assert not g.any()


@pytest.mark.parametrize("ragged,need_grad", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("K,N,M", [(1, 1, 1), (5, 31, 33), (3, 64, 64), (7, 65, 65), (2, 40, 130),
                                   (2, 400, 400)])
def test_overlap_evaluation(cuda, K, N, M, ragged, need_grad):
    from fast_shepherd_score_b200 import kernels as FK
    from oracle import align as oa
    d = _poses(K, N, M, K + N, ragged)
    g = {k: None if v is None else torch.as_tensor(v, device=cuda) for k, v in d.items()}
    common = dict(alpha=0.81, N_real=g["Nr"], M_real=g["Mr"], NEED_GRAD=need_grad)
    got = FK.overlap_score_grad_se3_batch(g["A"], g["B"], g["q"], g["t"], **common)
    _check(got, oa.overlap_grad(d["A"], d["B"], d["q"], d["t"], d["Nr"], d["Mr"], alpha=0.81),
           need_grad)
    got = FK.overlap_score_grad_esp_se3_batch(g["A"], g["B"], g["CA"], g["CB"], g["q"], g["t"],
                                              lam=0.3, **common)
    _check(got, oa.overlap_grad(d["A"], d["B"], d["q"], d["t"], d["Nr"], d["Mr"], alpha=0.81,
                                CA=d["CA"], CB=d["CB"], lam=0.3), need_grad)


@pytest.mark.parametrize("ragged,need_grad", [(False, True), (True, True), (True, False)])
@pytest.mark.parametrize("K,N,M", [(1, 1, 1), (5, 7, 9), (3, 33, 70), (2, 300, 40),
                                   (8191, 32, 32), (8190, 20, 11)])
def test_pharmacophore_evaluation(cuda, K, N, M, ragged, need_grad):
    from fast_shepherd_score_b200 import kernels as FK
    from oracle import align as oa
    d = _poses(K, N, M, K + N, ragged)
    g = {k: None if v is None else torch.as_tensor(v, device=cuda) for k, v in d.items()}
    got = FK.pharm_grad_dq_se3_batch(g["q"], g["t"], g["At"], g["Bt"], g["A"], g["B"], g["RV"],
                                     g["FV"], N_real=g["Nr"], M_real=g["Mr"],
                                     NEED_GRAD=need_grad)
    _check(got, oa.pharm_grad(d["A"], d["B"], d["RV"], d["FV"], d["At"], d["Bt"], d["q"], d["t"],
                              d["Nr"], d["Mr"]), need_grad)
