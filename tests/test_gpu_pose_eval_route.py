"""Pose evaluations on both sides of the batch size from which a pose of 65 to 255 fit points has one
warp instead of two, against the float64 oracle.  Tolerances as in test_gpu_kernels: values 1e-5,
gradients 1e-4 of the row's largest component or of the overlap, whose terms cancel in them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(9, 65), (20, 130), (5, 255), (5, 256)])
@pytest.mark.parametrize("more", [0, 1])
def test_overlap_evaluation_of_many_poses(cuda, N, M, more):
    from fast_shepherd_score_b200 import kernels as FK
    from oracle import align as oa
    K = 12 * torch.cuda.get_device_properties(cuda).multi_processor_count + more
    rng = np.random.default_rng(M + more)
    f = lambda *s, w=4.0: rng.uniform(-w, w, s).astype(np.float32)
    A, B, CA, CB, t = f(K, N, 3), f(K, M, 3), f(K, N, w=.3), f(K, M, w=.3), f(K, 3, w=1.0)
    q = rng.standard_normal((K, 4)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    Nr, Mr = (rng.integers(1, n + 1, K).astype(np.int32) for n in (N, M))
    g = lambda x: torch.as_tensor(x, device=cuda)
    got = FK.overlap_score_grad_esp_se3_batch(g(A), g(B), g(CA), g(CB), g(q), g(t), alpha=0.81,
                                              lam=0.3, N_real=g(Nr), M_real=g(Mr))
    V, dQ, dT = (x.cpu().numpy() for x in got)
    ref = oa.overlap_grad(A, B, q, t, Nr, Mr, alpha=0.81, CA=CA, CB=CB, lam=0.3)
    np.testing.assert_allclose(V, ref[0], rtol=1e-5, atol=1e-6)
    for x, r in ((dQ, ref[1]), (dT, ref[2])):
        scale = np.abs(r).max(1, keepdims=True) + np.abs(ref[0])[:, None] + 1e-2
        assert np.max(np.abs(x - r) / scale) < 1e-4
