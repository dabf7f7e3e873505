"""The two alignment kernels give the same bits for poses beyond the factored exponent's range, one
pair of a batch or many: molecules stretched to 31 A (some of a pose's point groups far, others
near), every remainder of a register tile, at 4 lanes both in the form for a few warps an SM and in
the form for many.  A fit molecule of more than 16 points per lane, unused, switches the kernel."""
import numpy as np
import pytest
import torch

from fast_shepherd_score_b200 import align as al
from fast_shepherd_score_b200.layout import CloudSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["shape", "esp", "esp_combo"])
@pytest.mark.parametrize("lanes,variant", [(4, 1), (4, 5), (8, 3), (8, 5), (16, 1), (32, 3)])
def test_far_rows_of_small_and_large_batches(cuda, mode, lanes, variant):
    if variant == 5 and mode == "esp_combo":
        variant = 1
    rng = np.random.default_rng(7)
    sizes = [1, lanes, *range(2 * lanes - 1, 14 * lanes, max(1, lanes * 3 // 4))]
    n, starts = len(sizes), 6
    stretch = np.linspace(0.6, 2.6, n)
    shape = lambda k, s: (rng.uniform(-6, 6, (k, 3)) * [s, 0.6, 0.6]).astype(np.float32)
    ref = [shape(int(k), s) for k, s in zip(rng.integers(3, 50, n), stretch)]
    fit = [shape(k, s) for k, s in zip(sizes, stretch[::-1])]
    q = lambda m: [(0.2 * rng.standard_normal(len(x))).astype(np.float32) for x in m]
    rq, fq = q(ref), q(fit)
    big = shape(16 * lanes + 1, 1.0)
    dev = lambda m, c: CloudSet.from_arrays(m, c, device=cuda)
    rs, fs = dev(ref, rq), dev(fit, fq)
    fb = dev(fit + [big], fq + q([big]))
    g = torch.Generator().manual_seed(5)
    sq = torch.nn.functional.normalize(torch.randn(n, starts, 4, generator=g), dim=-1).to(cuda)
    st = (2 * torch.randn(n, starts, 3, generator=g)).to(cuda)
    one, two = dict(fit=fs), dict(fit=fb)
    if mode == "esp_combo":
        surf = [shape(int(k), 1.0) for k in rng.integers(1, 60, 2 * n)]
        val = q(surf)
        rad = lambda m: torch.full((sum(map(len, m)),), 1.5, device=cuda)
        one.update(ref_atoms=rs, fit_atoms=fs, ref_radii=rad(ref), fit_radii=rad(fit),
                   ref_surf=dev(surf[:n], val[:n]), fit_surf=dev(surf[n:], val[n:]))
        two.update({**one, "fit": fb, "fit_atoms": fb, "fit_radii": rad(fit + [big]),
                    "fit_surf": dev(surf[n:] + surf[:1], val[n:] + val[:1])})

    def rows(repeat, kw):
        idx = torch.arange(n, dtype=torch.int32, device=cuda).repeat(repeat)
        rep = lambda x: x.repeat(repeat, 1, 1)
        out = al.align_packed(mode, ref=rs, pair_ref=idx, pair_fit=idx, seed_q=rep(sq),
                              seed_t=rep(st), steps=7, lr=0.1, lanes_per_pose=lanes,
                              kernel_variant=variant,
                              lam={"esp": 0.3, "esp_combo": 0.001}.get(mode), **kw).rows
        return torch.cat([x.reshape(repeat * n * starts, -1) for x in out], 1)

    few, other = rows(1, one), rows(1, two)
    assert torch.equal(few, other)
    # beyond four warps an SM: 148 SMs, at least one warp a pair and start block
    repeat = 4 * torch.cuda.get_device_properties(cuda).multi_processor_count // n + 2
    many, other = rows(repeat, one), rows(repeat, two)
    assert torch.equal(many, other)
    assert torch.equal(many, few.repeat(repeat, 1))


@pytest.mark.parametrize("kw", [{}, {"similarity": "tversky"}, {"similarity": "tversky_fit"},
                                {"pharm_extended": 1}, {"pharm_extended": 2}])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
def test_pharmacophore_rows_follow_one_lane(cuda, kw, lanes):
    """Mode "pharm" from 4 lanes a pose on against a lane a pose (the replicated state), three
    steps: scores are float32 sums of at most 400 Gaussians in another order (1e-6), which Adam's
    normalised step of 0.1 amplifies by up to 1e3 in components of small gradient: 1e-4 A a step."""
    from fast_shepherd_score_b200.layout import PharmSet
    rng = np.random.default_rng(8)
    counts = [1, 2, 3, 7, 8, 9, 15, 16, 17, 20, 31, 32, 33, 40]
    mk = lambda: PharmSet.from_arrays([rng.integers(0, 9, k) for k in counts],
                                      [rng.uniform(-4, 4, (k, 3)) for k in counts],
                                      [rng.standard_normal((k, 3)) for k in counts], device=cuda)
    ref, fit = mk(), mk()
    n, starts = len(counts), 10
    idx = torch.arange(n, dtype=torch.int32, device=cuda)
    g = torch.Generator().manual_seed(9)
    sq = torch.nn.functional.normalize(torch.randn(n, starts, 4, generator=g), dim=-1).to(cuda)
    st = torch.randn(n, starts, 3, generator=g).to(cuda)
    run = lambda lp, steps: al.align_packed("pharm", ref_ph=ref, fit_ph=fit, pair_ref=idx,
                                            pair_fit=idx, seed_q=sq, seed_t=st, steps=steps,
                                            lr=0.1, lanes_per_pose=lp, **kw).rows
    for steps, tol in ((1, 1e-5), (3, 2e-4)):
        a, b = run(lanes, steps), run(1, steps)
        torch.testing.assert_close(a[0], b[0], atol=tol, rtol=0)
    assert all(torch.isfinite(x).all() for x in a)
