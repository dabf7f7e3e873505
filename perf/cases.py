"""Workloads of the framework, as a user's program runs them, through its public entry points.

Families (``kind``):

* ``align``    -- multi-start alignment of a batch of molecule pairs whose clouds are on the GPU
  (``api.align_device``), or of host arrays (``api.align_host``) when ``host`` is set.  Batches of
  64 pairs or more name their tile (lanes per pose, code variant), as a program does that wants
  the same bits on every run and machine; smaller ones leave it to the library.
* ``poses``    -- overlap value and SE(3) gradient of many given poses, padded batches
  (``kernels.overlap_score_grad_se3_batch`` and its ESP and pharmacophore forms): one step of a
  caller's own pose optimiser.
* ``train``    -- differentiable Tanimoto scores of padded batches and their gradients
  (``autograd.get_overlap``, ``autograd.get_overlap_esp``).
* ``ragged``   -- the same of packed ragged sets, one query against many molecules
  (``autograd.tanimoto_packed``).
* ``library``  -- what is computed once per molecule or pair before an alignment: self overlaps
  and start poses.

Sizes are the framework's own workloads: 15-60 atoms, 3-20 pharmacophores, 200-400 surface
points, 8-50 starts, 30-200 Adam steps.  Atoms are uniform in a 6 A ball at least 1.2 A apart,
surfaces a jittered 5 A sphere with charges N(0, 0.1).
"""
import math

import numpy as np
import torch

from fast_shepherd_score_b200 import api, autograd, kernels, synthetic
from fast_shepherd_score_b200.layout import CloudSet, PharmSet

DEV = "cuda"
LAM = 0.3 * autograd.LAM_SCALING   # ESP width of surfaces, as the aligners scale it


def listed():
    return [
        # one molecule laid over another, host arrays in and out: an interactive call
        dict(name="align_pair", kind="align", mode="vol", pairs=1, lo=25, hi=35, starts=50,
             steps=200, lanes=0, variant=0, half=False, query=False, host=True),
        # plain shape alignment of a small batch (the 256-pair workload of the benchmark)
        dict(name="align_vol", kind="align", mode="vol", pairs=256, lo=15, hi=50, starts=50,
             steps=200, lanes=8, variant=3, half=False, query=False, host=False),
        # the ragged ESP surface workload of the benchmark, a quarter of its batch
        dict(name="align_surf_esp", kind="align", mode="surf_esp", pairs=1024, lo=200, hi=400,
             starts=50, steps=200, lanes=16, variant=3, half=False, query=False, host=False),
        # combined shape and pharmacophore batch of the benchmark, a quarter of its batch
        dict(name="align_vol_pharm", kind="align", mode="vol_pharm", pairs=4096, lo=15, hi=60,
             starts=50, steps=200, lanes=1, variant=0, half=False, query=False, host=False),
        # one query against a shard of a float16 library: what the screening server launches
        dict(name="screen_vol_pharm", kind="align", mode="vol_pharm", pairs=16384, lo=15, hi=60,
             starts=20, steps=100, lanes=8, variant=0, half=True, query=True, host=False),
        # pharmacophores alone, the mode's default starts and steps
        dict(name="align_pharm", kind="align", mode="pharm", pairs=1000, lo=15, hi=60, starts=32,
             steps=50, lanes=4, variant=0, half=False, query=False, host=False),
        # shape steered by atoms, scored with the surface ESP comparison, default starts and steps
        dict(name="align_combo", kind="align", mode="vol_and_surf_esp", pairs=512, lo=10, hi=25,
             starts=8, steps=60, lanes=16, variant=1, half=False, query=False, host=False),
        # one step of a caller's own optimiser: 256 pairs x 50 starts of atom clouds
        dict(name="poses_vol", kind="poses", mode="vol", poses=12800, lo=15, hi=50),
        # the same of ESP surfaces
        dict(name="poses_esp", kind="poses", mode="esp", poses=1600, lo=200, hi=400),
        # a training step's loss: 1024 generated molecules against one target, atoms and surface
        dict(name="train_1024", kind="train", batch=1024, atoms=60, surf=300, both=False),
        # one query scored in place against a ragged library, with coordinate gradients
        dict(name="ragged_20k", kind="ragged", mols=20000, lo=15, hi=60, esp=False),
        # a library taken in: self overlaps of both channels and start poses
        dict(name="library_100k", kind="library", mols=100000, lo=15, hi=60, starts=20,
             half=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


TERMS = 8e11   # pair terms of the largest drawn alignment, below the largest listed one's


def draw(rng):
    kind = rng.choice(["align", "align", "align", "poses", "train", "ragged", "library"])
    if kind == "align":
        mode = rng.choice(["vol", "vol_esp", "surf", "surf_esp", "vol_pharm", "vol_color", "pharm",
                           "vol_and_surf_esp"])
        starts, steps = rng.randint(8, 50), rng.randint(30, 200)
        surf = mode in ("surf", "surf_esp")
        lo = rng.randint(200, 300) if surf else 10 if mode == "vol_and_surf_esp" else 15
        hi = rng.randint(lo, 400) if surf else 25 if mode == "vol_and_surf_esp" else \
            rng.randint(30, 60)
        most = TERMS / (starts * steps * ((lo + hi) / 2) ** 2)
        pairs = _log(rng, 1, max(1, min(16384 if mode != "vol_and_surf_esp" else 600, most)))
        lanes = variant = 0
        if pairs >= 64:
            lanes = {"vol": rng.choice([4, 8]), "vol_esp": 8, "surf": 16, "surf_esp": 16,
                     "pharm": rng.choice([1, 4]), "vol_and_surf_esp": 16}.get(
                         mode, rng.choice([1, 4, 8]))
            variant = {"vol": rng.choice([1, 3, 5]), "vol_esp": 3, "surf": rng.choice([3, 4]),
                       "surf_esp": rng.choice([3, 4]), "vol_and_surf_esp": 1}.get(mode, 0)
        half = mode not in ("pharm", "vol_and_surf_esp") and rng.random() < 0.5
        return dict(kind=kind, mode=mode, pairs=pairs, lo=lo, hi=hi, starts=starts, steps=steps,
                    lanes=lanes, variant=variant, half=half, query=rng.random() < 0.5,
                    host=False)
    if kind == "poses":
        mode = rng.choice(["vol", "esp", "pharm"])
        if mode == "esp":
            lo = rng.randint(150, 300)
            return dict(kind=kind, mode=mode, poses=_log(rng, 8, 1600), lo=lo,
                        hi=rng.randint(lo, 400))
        lo, hi = (15, rng.randint(30, 60)) if mode == "vol" else (3, rng.randint(10, 20))
        return dict(kind=kind, mode=mode, poses=_log(rng, 50, 13000), lo=lo, hi=hi)
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 1, 1024), atoms=rng.randint(15, 60),
                    surf=rng.randint(100, 400), both=rng.random() < 0.5)
    if kind == "ragged":
        esp = rng.random() < 0.5
        lo, hi = (100, rng.randint(200, 400)) if esp else (15, rng.randint(30, 60))
        return dict(kind=kind, mols=_log(rng, 30, 1000 if esp else 20000), lo=lo, hi=hi, esp=esp)
    return dict(kind=kind, mols=_log(rng, 100, 100000), lo=15, hi=rng.randint(30, 60),
                starts=rng.randint(5, 50), half=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _gen(seed, k):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 16 + k)
    return g


def _set(pts, counts):
    off = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(counts, out=off[1:])
    return CloudSet(pts, torch.from_numpy(off.astype(np.int32)).to(DEV), counts,
                    int(counts.max()))


def _counts(g, n, lo, hi):
    return torch.randint(lo, hi + 1, (n,), generator=g, device=DEV)


def _sphere(g, n):
    """n surface points with charges, (n, 4)."""
    u = torch.randn(n, 3, generator=g, device=DEV)
    p = 5.0 * u / u.norm(dim=1, keepdim=True) + 0.3 * torch.randn(n, 3, generator=g, device=DEV)
    return torch.cat([p, 0.1 * torch.randn(n, 1, generator=g, device=DEV)], 1)


def _surfaces(seed, k, n, lo, hi):
    g = _gen(seed, k)
    counts = _counts(g, n, lo, hi).cpu().numpy().astype(np.int64)
    return _set(_sphere(g, int(counts.sum())), counts)


def _molecules(seed, k, n, lo, hi, charged=False):
    atoms, ph = synthetic.library_on_device(n, seed=int(seed) * 16 + k, device=DEV, atom_lo=lo,
                                            atom_hi=hi)
    if charged:
        atoms.pts[:, 3] = 0.2 * torch.randn(atoms.pts.shape[0], generator=_gen(seed, k + 8),
                                            device=DEV)
    return atoms, ph


def _halved(atoms, ph):
    """The set in float16, as a library read from a float16 store is kept on the device."""
    atoms = CloudSet(atoms.pts.half(), atoms.off, atoms.counts, atoms.max_points)
    if ph is not None:
        anc = ph.anc.half()
        anc[:, 3] = ph.anc[:, 3].contiguous().view(torch.int32).half()
        ph = PharmSet(anc, ph.vec.half(), ph.off, ph.counts, ph.max_points)
    return atoms, ph


def _combo(mols):
    return (CloudSet.from_arrays([m["centers"] for m in mols], device=DEV),
            CloudSet.from_arrays([m["atoms"] for m in mols], [m["charges"] for m in mols],
                                 device=DEV),
            torch.from_numpy(np.concatenate([m["radii"] for m in mols])).to(DEV),
            CloudSet.from_arrays([m["surf"] for m in mols], [m["surf_esp"] for m in mols],
                                 device=DEV))


def _prepare_align(case, seed):
    P, lo, hi, mode = case["pairs"], case["lo"], case["hi"], case["mode"]
    n_ref = 1 if case["query"] else P
    r_lo, r_hi = (lo, hi)
    if case["query"]:   # a query of middling size: the work does not hang on the seed
        r_lo = r_hi = (lo + hi) // 2
    kw = dict(num_seeds=case["starts"], steps=case["steps"], lr=0.1)
    if case["lanes"]:
        kw.update(lanes_per_pose=case["lanes"], kernel_variant=case["variant"])
    rp = fp = None
    if mode == "vol_and_surf_esp":
        rng = np.random.default_rng(seed)
        mk = lambda n, a, b: _combo(synthetic.esp_combo_molecules(n, rng, heavy_lo=a,
                                                                  heavy_hi=b))
        (rc, ra, rr, rs), (fc, fa, fr, fs) = mk(n_ref, r_lo, r_hi), mk(P, lo, hi)
        kw.update(lam=0.001, ref_atoms=ra, ref_radii=rr, ref_surf=rs, fit_atoms=fa, fit_radii=fr,
                  fit_surf=fs)
    elif mode in ("surf", "surf_esp"):
        rc, fc = _surfaces(seed, 0, n_ref, r_lo, r_hi), _surfaces(seed, 1, P, lo, hi)
        kw.update(alpha=1.216, lam=0.3)
    else:
        esp = mode == "vol_esp"
        rc, rp = _molecules(seed, 0, n_ref, r_lo, r_hi, esp)
        fc, fp = _molecules(seed, 1, P, lo, hi, esp)
        kw.update(lam=0.3)
    if mode in ("vol", "vol_esp", "surf", "surf_esp", "vol_and_surf_esp"):
        rp = fp = None
    if mode == "pharm":
        rc = fc = None
    if case["half"]:
        fc, fp = _halved(fc, fp)
    if case["host"]:
        host = lambda cs: api.HostBatch(cs.pts.cpu().numpy(), cs.counts)
        return dict(mode=mode, host=(host(rc), host(fc)), kw=kw)
    pf = torch.arange(P, dtype=torch.int32, device=DEV)
    pr = torch.zeros_like(pf) if case["query"] else pf
    return dict(mode=mode, sets=(rc, fc, rp, fp), pairs=(pr, pf), kw=kw)


def _padded(g, points, counts):
    """Rows of `points` (n, pad, .) beyond each count zeroed, as a padded batch has them."""
    mask = torch.arange(points.shape[1], device=DEV)[None] < counts[:, None]
    return torch.where(mask[..., None], points, torch.zeros_like(points))


def _ball(g, n, pad, radius=6.0):
    v = torch.randn(n, pad, 3, generator=g, device=DEV)
    r = radius * torch.rand(n, pad, 1, generator=g, device=DEV) ** (1 / 3)
    return r * v / v.norm(dim=-1, keepdim=True)


def _prepare_poses(case, seed):
    g, K, lo, hi = _gen(seed, 2), case["poses"], case["lo"], case["hi"]
    n, m = _counts(g, K, lo, hi), _counts(g, K, lo, hi)
    s = dict(mode=case["mode"], N=n.int(), M=m.int())
    pad_n, pad_m = int(n.max()), int(m.max())
    if case["mode"] == "esp":
        A = _sphere(g, K * pad_n).view(K, pad_n, 4)
        B = _sphere(g, K * pad_m).view(K, pad_m, 4)
        s.update(CA=A[..., 3].contiguous(), CB=B[..., 3].contiguous())
        A, B = A[..., :3], B[..., :3]
    else:
        A, B = _ball(g, K, pad_n), _ball(g, K, pad_m)
    if case["mode"] == "pharm":
        unit = lambda p: torch.nn.functional.normalize(
            torch.randn(K, p, 3, generator=g, device=DEV), dim=-1)
        s.update(TA=torch.randint(0, 8, (K, pad_n), generator=g, device=DEV, dtype=torch.int32),
                 TB=torch.randint(0, 8, (K, pad_m), generator=g, device=DEV, dtype=torch.int32),
                 VA=unit(pad_n), VB=unit(pad_m))
    s.update(A=_padded(g, A, n).contiguous(), B=_padded(g, B, m).contiguous())
    s["q"] = torch.nn.functional.normalize(torch.randn(K, 4, generator=g, device=DEV), dim=1)
    s["t"] = 0.5 * torch.randn(K, 3, generator=g, device=DEV)
    return s


def _prepare_train(case, seed):
    g, B = _gen(seed, 3), case["batch"]
    T = B if case["both"] else 1   # targets of their own (both sides differentiated), or one
    surf = lambda n: _sphere(g, n * case["surf"]).view(n, case["surf"], 4)
    s, ts = surf(B), surf(T)
    leaf = lambda x, on=True: x.contiguous().requires_grad_(on)
    return dict(atoms=leaf(_ball(g, B, case["atoms"])), surf=leaf(s[..., :3]),
                charge=leaf(s[..., 3]), t_atoms=leaf(_ball(g, T, case["atoms"]), case["both"]),
                t_surf=leaf(ts[..., :3], case["both"]), t_charge=leaf(ts[..., 3], case["both"]))


def _prepare_ragged(case, seed):
    n, lo, hi = case["mols"], case["lo"], case["hi"]
    make = (lambda k, m: _surfaces(seed, k, m, hi, hi)) if case["esp"] else \
        (lambda k, m: _molecules(seed, k, m, hi, hi)[0])
    ref, fit = make(5, 1), make(4, n)
    # each molecule keeps its first few points: sizes spread over [lo, hi], the same every time
    counts = lo + np.random.default_rng(n).permutation(n) % (hi - lo + 1)
    keep = torch.arange(hi, device=DEV)[None] < torch.from_numpy(counts).to(DEV)[:, None]
    fit = _set(fit.pts.view(n, hi, 4)[keep], counts)
    pf = torch.arange(n, dtype=torch.int32, device=DEV)
    return dict(ref=ref, fit=fit, pf=pf, pr=torch.zeros_like(pf), pts=fit.pts.requires_grad_(),
                lam=LAM if case["esp"] else None, weight=torch.ones(n, device=DEV))


def _prepare_library(case, seed):
    n = case["mols"]
    atoms, ph = _molecules(seed, 6, n, case["lo"], case["hi"])
    query = _molecules(seed, 7, 1, case["hi"], case["hi"])[0]
    if case["half"]:
        atoms, ph = _halved(atoms, ph)
    pf = torch.arange(n, dtype=torch.int32, device=DEV)
    return dict(atoms=atoms, ph=ph, query=query, pf=pf, pr=torch.zeros_like(pf),
                starts=case["starts"])


def prepare(case, seed):
    s = {"align": _prepare_align, "poses": _prepare_poses, "train": _prepare_train,
         "ragged": _prepare_ragged, "library": _prepare_library}[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "align":
        if "host" in s:
            out = api.align_host(s["mode"], *s["host"], device=DEV, **s["kw"])
            return out.scores, out.q, out.t
        rc, fc, rp, fp = s["sets"]
        score, q, t = api.align_device(s["mode"], rc, fc, rp, fp, *s["pairs"], **s["kw"])
        return score, q, t
    if kind == "poses":
        common = dict(N_real=s["N"], M_real=s["M"])
        if s["mode"] == "vol":
            return kernels.overlap_score_grad_se3_batch(s["A"], s["B"], s["q"], s["t"], **common)
        if s["mode"] == "esp":
            return kernels.overlap_score_grad_esp_se3_batch(s["A"], s["B"], s["CA"], s["CB"],
                                                            s["q"], s["t"], lam=LAM, **common)
        return kernels.pharm_grad_dq_se3_batch(s["q"], s["t"], s["TA"], s["TB"], s["A"], s["B"],
                                               s["VA"], s["VB"], **common)
    if kind == "train":
        leaves = [s[k] for k in ("atoms", "surf", "charge", "t_atoms", "t_surf", "t_charge")
                  if s[k].requires_grad]
        vol = autograd.get_overlap(s["t_atoms"], s["atoms"])
        esp = autograd.get_overlap_esp(s["t_surf"], s["surf"], s["t_charge"], s["charge"],
                                       alpha=1.216, lam=LAM)
        grads = torch.autograd.grad(vol.sum() + esp.sum(), leaves)
        return (vol.detach(), esp.detach()) + grads
    if kind == "ragged":
        score = autograd.tanimoto_packed(s["ref"].pts, s["ref"].off, s["pts"], s["fit"].off,
                                         s["pr"], s["pf"], lam=s["lam"],
                                         max_ref=s["ref"].max_points,
                                         max_fit=s["fit"].max_points)
        grad, = torch.autograd.grad(score, s["pts"], s["weight"])
        return score.detach(), grad
    shape = kernels.self_overlap(s["atoms"], 0.81)
    pharm = kernels.pharm_self_overlap(s["ph"])
    q, t = kernels.seeds(s["query"], s["atoms"], s["pr"], s["pf"], s["starts"])
    return shape, pharm, q, t


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    """Bytes of every input and output once; per pair of points the multiply-adds of its
    exponent and sums (7 for a shape gradient term, 8 with charges, 4 for a value), two
    operations each."""
    kind = case["kind"]
    mean = (case["lo"] + case["hi"]) / 2 if "lo" in case else 0
    if kind == "align":
        P, mode = case["pairs"], case["mode"]
        poses = P * case["starts"] * case["steps"]
        point = 8 if case["half"] else 16
        mols = P + (1 if case["query"] else P)
        size = 11.5 * 2 if mode == "pharm" else mean
        if mode in ("vol_pharm", "vol_color"):
            size = mean + 2 * 11.5
        if mode == "vol_and_surf_esp":
            size = mean + 1.8 * mean * 1.25 + 150
        terms = 0.0 if mode == "pharm" else mean ** 2 * (16 if "esp" in mode else 14)
        if mode in ("pharm", "vol_pharm", "vol_color"):
            terms += 11.5 ** 2 / 8 * 24
        if mode == "vol_and_surf_esp":
            terms = mean ** 2 * 14 + 2 * 150 * 1.8 * mean * 12
        return dict(bytes=mols * size * point + 32 * P, flops=poses * terms)
    if kind == "poses":
        K, per = case["poses"], {"vol": 12, "esp": 16, "pharm": 28}[case["mode"]]
        terms = mean ** 2 * (16 if case["mode"] == "esp" else 14)
        if case["mode"] == "pharm":
            terms = mean ** 2 / 8 * 24
        return dict(bytes=K * (2 * mean * per + 28 + 8 + 32), flops=K * terms)
    if kind == "train":
        B, n, m = case["batch"], case["atoms"], case["surf"]
        sides = 2 if case["both"] else 1
        # cross terms with gradients, the own cloud's with gradients where it is differentiated,
        # values of half the own pairs where it is not
        t_a = n * n * (14 * (1 + sides) + (0 if case["both"] else 4 / B))
        t_s = m * m * (16 * (1 + sides) + (0 if case["both"] else 5 / B))
        size = (12 * n + 16 * m) * (B + (B if case["both"] else 1))
        grads = (12 * n + 16 * m) * B * sides
        return dict(bytes=size + grads + 8 * B, flops=B * (t_a + t_s))
    if kind == "ragged":
        K, c = case["mols"], 16 if case["esp"] else 14
        return dict(bytes=K * mean * 32 + 8 * K, flops=K * (case["hi"] * mean + mean ** 2) * c)
    K = case["mols"]
    point = 8 if case["half"] else 16
    return dict(bytes=K * (mean * point * 2 + 2 * 11.5 * point + 8 + 28 * case["starts"]),
                flops=K * (mean ** 2 * 4 + 11.5 ** 2 / 16 * 20 + 30 * mean))


# ---------------------------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------------------------
def _const(alpha):
    return math.pi ** 1.5 / (2 * alpha) ** 1.5


def _overlap64(x, y, alpha, mask=None, cx=None, cy=None, lam=None):
    """sum_ij exp(-alpha/2 |x_i - y_j|^2) [exp(-(c_i - c_j)^2 / lam)] per batch row, (B, n, 3)."""
    e = -0.5 * alpha * ((x[:, :, None] - y[:, None]) ** 2).sum(-1)
    if cx is not None:
        e = e - (cx[:, :, None] - cy[:, None]) ** 2 / lam
    g = torch.exp(e)
    if mask is not None:
        g = g * mask
    return _const(alpha) * g.sum((1, 2))


def _rot64(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)],
                       -1).reshape(q.shape[:-1] + (3, 3))


_ALPHA = (1.0, 1.0, 0.7, 0.7, 1.0, 1.0, 1.0, 1.0, 1.0)   # Gaussian widths of the types
_CLASS = (1, 1, 2, 0, 1, 0, 0, 0, 3)                     # plain, directed, aromatic, dummy


def _pharm64(x, y, u, v, tx, ty, mask):
    """Typed directional overlap per batch row: same-type anchors, weight (2 + cos) / 3."""
    al = torch.tensor(_ALPHA, device=x.device, dtype=torch.float64)[tx.long()][:, :, None]
    cls = torch.tensor(_CLASS, device=x.device)[tx.long()][:, :, None]
    g = (math.pi / (2 * al)) ** 1.5 * torch.exp(
        -0.5 * al * ((x[:, :, None] - y[:, None]) ** 2).sum(-1))
    cos = (u[:, :, None] * v[:, None]).sum(-1)
    one = torch.ones_like(cos)
    w = torch.where(cls == 1, (cos.clamp(0, 1) + 2) / 3,
                    torch.where(cls == 2, (cos.abs() + 2) / 3, one))
    same = (tx[:, :, None] == ty[:, None]) & (cls != 3) & mask
    return (g * w * same).sum((1, 2))


def _exact_poses(case, seed):
    s = _prepare_poses(case, seed)
    out = []
    step = max(1, int(2e7 // (s["A"].shape[1] * s["B"].shape[1])))
    for a in range(0, case["poses"], step):
        c = {k: v[a:a + step].double() for k, v in s.items() if isinstance(v, torch.Tensor)}
        q, t = c["q"].requires_grad_(), c["t"].requires_grad_()
        R = _rot64(q)
        y = c["B"] @ R.transpose(1, 2) + t[:, None]
        at = lambda k, n: torch.arange(c[k].shape[1], device=DEV)[None] < n[:, None]
        mask = at("A", c["N"])[:, :, None] & at("B", c["M"])[:, None]
        if case["mode"] == "pharm":
            unit = lambda v: v / v.norm(dim=-1, keepdim=True).clamp(min=1e-12)
            V = _pharm64(c["A"], y, unit(c["VA"]), unit(c["VB"]) @ R.transpose(1, 2), c["TA"],
                         c["TB"], mask)
        else:
            V = _overlap64(c["A"], y, 0.81, mask, c.get("CA"), c.get("CB"), LAM)
        out.append((V.detach(),) + torch.autograd.grad(V.sum(), (q, t)))
    return tuple(torch.cat(x) for x in zip(*out))


def _tanimoto64(x, y, alpha, **kw):
    ab = _overlap64(x, y, alpha, **kw)
    own = lambda p, c: _overlap64(p, p, alpha, **({} if "cx" not in kw else
                                                  dict(cx=c, cy=c, lam=kw["lam"])))
    return ab / (own(x, kw.get("cx")) + own(y, kw.get("cy")) - ab)


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    names = ("atoms", "surf", "charge", "t_atoms", "t_surf", "t_charge")
    keep = [k for k in names if s[k].requires_grad]
    out = []
    step = max(1, int(2e7 // case["surf"] ** 2))
    for a in range(0, case["batch"], step):
        c = {k: (s[k] if s[k].shape[0] == 1 < case["batch"] else s[k][a:a + step]).detach()
             .double().requires_grad_(k in keep) for k in names}
        n = c["atoms"].shape[0]
        full = {k: v.expand((n,) + v.shape[1:]) for k, v in c.items()}
        vol = _tanimoto64(full["t_atoms"], full["atoms"], 0.81)
        esp = _tanimoto64(full["t_surf"], full["surf"], 1.216, cx=full["t_charge"],
                          cy=full["charge"], lam=LAM)
        out.append((vol.detach(), esp.detach())
                   + torch.autograd.grad(vol.sum() + esp.sum(), [c[k] for k in keep]))
    return tuple(torch.cat(x) for x in zip(*out))


def _rows(cs, pts):
    """(n, max, 4) float64 padded form of a packed set, and its mask."""
    n = (cs.off[1:] - cs.off[:-1]).long()
    ar = torch.arange(cs.max_points, device=DEV)[None]
    mask = ar < n[:, None]
    idx = torch.where(mask, cs.off[:-1].long()[:, None] + ar, torch.zeros_like(ar))
    return pts.detach().double()[idx] * mask[..., None], mask, idx


def _exact_ragged(case, seed):
    s = _prepare_ragged(case, seed)
    ref = s["ref"].pts.double()[None]
    rows, mask, idx = _rows(s["fit"], s["pts"])
    kw = lambda a, b: dict(cx=a[..., 3], cy=b[..., 3], lam=s["lam"]) if case["esp"] else {}
    aa = _overlap64(ref[..., :3], ref[..., :3], 0.81, **kw(ref, ref))
    score = torch.empty(case["mols"], dtype=torch.float64, device=DEV)
    grad = torch.zeros(s["pts"].shape, dtype=torch.float64, device=DEV)
    step = max(1, int(2e7 // (rows.shape[1] ** 2)))
    for a in range(0, case["mols"], step):
        x, m = rows[a:a + step].requires_grad_(), mask[a:a + step]
        r = ref.expand(x.shape[0], -1, -1)
        ab = _overlap64(r[..., :3], x[..., :3], 0.81, m[:, None, :], **kw(r, x))
        bb = _overlap64(x[..., :3], x[..., :3], 0.81, m[:, :, None] & m[:, None, :], **kw(x, x))
        sc = ab / (aa + bb - ab)
        score[a:a + step] = sc.detach()
        gx, = torch.autograd.grad(sc.sum(), x)
        grad[idx[a:a + step][m]] = gx[m]
    return score, grad


def _exact_library(case, seed):
    s = _prepare_library(case, seed)
    rows, mask, _ = _rows(s["atoms"], s["atoms"].pts)
    anc, am, idx = _rows(s["ph"], s["ph"].anc)
    word = s["ph"].anc[:, 3].contiguous()
    types = (word.long() if case["half"] else word.view(torch.int32).long())[idx]
    vec = _rows(s["ph"], s["ph"].vec)[0][..., :3]
    vec = vec / vec.norm(dim=-1, keepdim=True).clamp(min=1e-12)
    shape, pharm = [], []
    for a in range(0, case["mols"], 4000):
        x, m = rows[a:a + 4000, :, :3], mask[a:a + 4000]
        shape.append(_overlap64(x, x, 0.81, m[:, :, None] & m[:, None, :]))
        x, v, t, m = (z[a:a + 4000] for z in (anc[..., :3], vec, types, am))
        pharm.append(_pharm64(x, x, v, v, t, t, m[:, :, None] & m[:, None, :]))
    return torch.cat(shape), torch.cat(pharm), None, None


def exact(case, seed):
    # an alignment is a long chaotic iteration: rounding decides which optimum a start ends in,
    # so it has no 64-bit value to be near to
    fn = {"poses": _exact_poses, "train": _exact_train, "ragged": _exact_ragged,
          "library": _exact_library}.get(case["kind"])
    return None if fn is None else fn(case, seed)
