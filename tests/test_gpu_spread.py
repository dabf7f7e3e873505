"""The kernel that spreads a pose's optimiser state over its lanes gives the bits of the one that
replicates it.  A launch whose largest fit molecule has more than 16 points per lane runs on the
latter, so an unused large molecule in the set switches kernels for the same pairs: every
remainder of the register tiles (points per lane 1, 2, ...), empty clouds, poses beyond the
factored exponent's range, both channels and the ESP comparison."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200 import kernels as K
from fast_shepherd_score_b200 import synthetic as syn
from fast_shepherd_score_b200.layout import CloudSet, PharmSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["shape", "esp", "shape_pharm", "shape_color", "esp_combo"])
@pytest.mark.parametrize("lanes,variant", [(4, 1), (8, 3), (8, 5), (16, 3), (32, 3)])
def test_rows_equal_replicated_state(cuda, mode, lanes, variant):
    if variant != 1 and mode in ("shape_pharm", "shape_color"):
        variant = 1
    if variant == 5 and mode == "esp_combo":
        pytest.skip("no such variant")
    rng = np.random.default_rng(12)
    sizes = list(range(0, 12 * lanes, max(1, lanes // 4))) if lanes < 32 else [0, 1, 33, 200, 500]
    n = len(sizes)
    cloud = lambda k: (3.0 * rng.standard_normal((k, 3))).astype(np.float32)
    charge = lambda k: (0.2 * rng.standard_normal(k)).astype(np.float32)
    ref = [cloud(int(k)) for k in rng.integers(3, 50, n)]
    fit, big = [cloud(k) for k in sizes], cloud(16 * lanes + 1)
    rq, fq, bq = [charge(len(x)) for x in ref], [charge(k) for k in sizes], charge(len(big))
    small = lambda pts, q: CloudSet.from_arrays(pts, q, device=cuda)
    idx = torch.arange(n, dtype=torch.int32, device=cuda)
    rs, fs, fb = small(ref, rq), small(fit, fq), small(fit + [big], fq + [bq])
    sq, st = K.seeds(rs, fs, idx, idx, 13)
    st[:, ::4] += torch.tensor([13.0, 0.0, 0.0], device=cuda)   # some start far off
    kw = dict(ref=rs, pair_ref=idx, pair_fit=idx, seed_q=sq, seed_t=st, steps=9, lr=0.1,
              lanes_per_pose=lanes, kernel_variant=variant,
              lam={"esp": 0.3, "esp_combo": 0.001}.get(mode))
    one, two = dict(kw, fit=fs), dict(kw, fit=fb)
    if "_" in mode and mode != "esp_combo":
        ph = syn.pharm_features(rng, [np.concatenate([x, np.zeros((1, 3), np.float32)])
                                      for x in ref + fit], rng.integers(0, 40, 2 * n))
        mk = lambda f: PharmSet.from_arrays([x[0] for x in f], [x[1] for x in f],
                                            [x[2] for x in f], device=cuda)
        one.update(ref_ph=mk(ph[:n]), fit_ph=mk(ph[n:]))
        two.update(ref_ph=one["ref_ph"], fit_ph=mk(ph[n:] + [ph[0]]))
    if mode == "esp_combo":
        surf = [5.0 + cloud(int(k)) for k in rng.integers(1, 90, 2 * n + 1)]
        val = [charge(len(s)) for s in surf]
        rad = lambda m: torch.full((sum(len(x) for x in m),), 1.5, device=cuda)
        one.update(ref_atoms=rs, fit_atoms=fs, ref_radii=rad(ref), fit_radii=rad(fit),
                   ref_surf=small(surf[:n], val[:n]), fit_surf=small(surf[n:-1], val[n:-1]))
        two.update(one, fit=fb, fit_atoms=fb, fit_radii=rad(fit + [big]),
                   fit_surf=small(surf[n:], val[n:]))
    a, b = al.align_packed(mode, **one).rows, al.align_packed(mode, **two).rows
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.cpu().numpy(), y.cpu().numpy())
