"""vol_and_surf_esp launches whose CTAs would all be resident, unevenly, leave the extra ones for the
SMs that are done first: rows are the bits of a launch with one CTA an SM, on both sides of the rule
(CTAs an SM times 100; lanes)."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200.layout import CloudSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm,lanes", [(199, 16), (200, 16), (201, 16), (249, 16), (251, 16), (399, 16),
                                          (401, 16), (401, 8), (450, 8), (799, 8), (1390, 4)])
def test_rows_do_not_depend_on_resident_ctas(cuda, per_sm, lanes):
    P = torch.cuda.get_device_properties(cuda).multi_processor_count * per_sm // 100
    rng = np.random.default_rng(per_sm)
    n, starts = 40, 8
    cloud = lambda lo, hi, w: [rng.uniform(-w, w, (k, 3)).astype(np.float32)
                               for k in rng.integers(lo, hi, n)]
    dev = lambda m: CloudSet.from_arrays(m, [(0.2 * rng.standard_normal(len(x))).astype(np.float32)
                                             for x in m], device=cuda)
    rad = lambda m: torch.full((sum(map(len, m)),), 1.5, device=cuda)
    ra, fa = cloud(10, 30, 3.0), cloud(10, 30, 3.0)
    kw = dict(ref=dev(cloud(5, 12, 3.0)), fit=dev(cloud(5, 12, 3.0)), ref_atoms=dev(ra),
              fit_atoms=dev(fa), ref_radii=rad(ra), fit_radii=rad(fa),
              ref_surf=dev(cloud(20, 60, 5.0)), fit_surf=dev(cloud(20, 60, 5.0)), lam=0.001)
    i = torch.arange(P, device=cuda)
    g = torch.Generator().manual_seed(1)
    q = torch.nn.functional.normalize(torch.randn(P, starts, 4, generator=g), dim=-1).to(cuda)
    t = torch.randn(P, starts, 3, generator=g).to(cuda)
    run = lambda cps: al.align_packed("esp_combo", pair_ref=i % n, pair_fit=(3 * i) % n, seed_q=q,
                                      seed_t=t, steps=8, lr=0.1, lanes_per_pose=lanes, chunks=1,
                                      kernel_variant=1, cta_per_sm=cps, **kw).rows
    for a, b in zip(run(0), run(1)):
        assert torch.equal(a, b)
