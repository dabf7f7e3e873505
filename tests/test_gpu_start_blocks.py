"""The library's choice of start blocks (chunks = 0) changes no result: rows equal those of one
start per block, for a pair alone (one-warp CTAs over the SMs), a launch of less than two rounds
of CTAs, several rounds (the residency rule), and short runs."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200 import kernels as K
from fast_shepherd_score_b200 import synthetic as syn
from fast_shepherd_score_b200.layout import CloudSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,starts,steps", [(1, 50, 20), (1, 5, 20), (300, 20, 8),
                                                (4000, 13, 8), (300, 20, 7)])
@pytest.mark.parametrize("lanes", [1, 4, 16, 32])
def test_rows_equal_single_start_blocks(cuda, pairs, starts, steps, lanes):
    refs, fits = syn.shape_pairs(min(pairs, 300), seed=5, lo=15, hi=40)
    ref, fit = (CloudSet.from_arrays(m, device=cuda) for m in (refs, fits))
    idx = torch.arange(pairs, dtype=torch.int32, device=cuda) % len(refs)
    sq, st = K.seeds(ref, fit, idx, idx, starts)
    kw = dict(ref=ref, fit=fit, pair_ref=idx, pair_fit=idx, seed_q=sq, seed_t=st, steps=steps,
              lr=0.1, lanes_per_pose=lanes, kernel_variant=3)
    auto = al.align_packed("shape", **kw).rows
    one = al.align_packed("shape", chunks=starts, **kw).rows
    for a, b in zip(auto, one):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
