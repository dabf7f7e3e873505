"""No start block without a start is launched: a CTA's whole warps hold more poses than
ceil(starts / chunks) when that many lanes do not fill them, so fewer blocks are left.  Every CTA takes
a work item more than there are (the one that ends it), so with one CTA per block the work counter
ends at twice the blocks."""
import pytest
import torch

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200.layout import CloudSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,chunks,blocks", [(8, 26, 13), (8, 13, 13), (1, 50, 2), (4, 9, 7),
                                                 (16, 25, 25), (16, 50, 25), (32, 50, 50), (2, 1, 1)])
def test_blocks_launched(cuda, lanes, chunks, blocks):
    g = torch.Generator().manual_seed(1)
    cloud = CloudSet.from_arrays([torch.randn(20, 3, generator=g).numpy()], device=cuda)
    one = torch.zeros(1, dtype=torch.int32, device=cuda)
    q = torch.nn.functional.normalize(torch.randn(1, 50, 4, generator=g), dim=-1).to(cuda)
    t = torch.randn(1, 50, 3, generator=g).to(cuda)
    scratch = torch.zeros(2, dtype=torch.int32, device=cuda)
    kw = dict(ref=cloud, fit=cloud, pair_ref=one, pair_fit=one, seed_q=q, seed_t=t, steps=10,
              lr=0.1, lanes_per_pose=lanes, kernel_variant=1)
    rows = al.align_packed("shape", chunks=chunks, scratch=scratch, **kw).rows
    assert scratch.tolist() == [2 * blocks, 0]
    for x, y in zip(rows, al.align_packed("shape", chunks=50, **kw).rows):
        assert torch.equal(x, y)
