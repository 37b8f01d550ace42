"""The work that users of this package have it do, as measurable cases.

Phase tables are the repository's own fixtures (``tests/golden``): FEFF's native mesh of about 60 real-axis energies, or
the same tables resampled to a uniform k grid (the batched stage's benchmark form).  Path lists are what the path finder
returns for seeded structures of the repository's workloads -- a random Fe/O/Pt packing, an fcc Cu cluster, thermal bcc
Fe, disordered rock-salt NiO -- enumerated here with plain torch: every path of 2..legs legs of half length <= rmax, in
the finder's order (grouped by leg count), the smaller of a sequence and its reverse kept with degeneracy 2, and
coordinates relative to the absorber in FP32 as the finder leaves them.  A case's structure and path list are its own;
the seed moves the atoms (0.03 A), as a trajectory or a refinement does between two enumerations.

``exact`` is the path stage restated in complex128 torch (its derivatives by autograd).
"""
import math
from pathlib import Path

import numpy as np
import torch

GOLDEN = Path(__file__).resolve().parent.parent / "tests" / "golden"
BOHR = 0.52917721067
NK = 401
PHASE = {"packing": "cfg2_phase", "cu": "cfg1_cu", "bcc": "cfg4_fe_phase", "nio": "cfg5_nik_phase", "l3": "case_A014"}


def listed():
    return [
        # one spectrum of a crystal through the drop-in stage: per leg count cchi -> chi_fine -> weighted sum, as the
        # reference's chain.run does; a few hundred paths on FEFF's native mesh (the smallest call, latency)
        dict(name="dropin_cu", kind="dropin", struct="cu", rmax=4.5, legs=4, nk=0, fp64=False, take=400),
        # the same front end in the plain FP64 form on one of its 4096-path chunks of longer paths, resampled tables
        dict(name="dropin_fp64_chunk", kind="dropin", struct="packing", rmax=6.9, legs=5, nk=401, fp64=True, take=4096),
        # a refinement's forward model through the drop-in stage: signal, fine grid and the gradient of every
        # coordinate (the reference's PathSpectra), a chunk of its paths
        dict(name="dropin_grad", kind="dropin_grad", struct="packing", rmax=6.6, legs=4, nk=0, fp64=False, take=2048),
        # one structure's fit: a few hundred paths, one fused call with its gradient (a step of a small refinement)
        dict(name="fused_fit_small", kind="fused_grad", struct="packing", rmax=5.4, legs=4, nk=0, fp64=False, absorbers=1),
        # an L3 edge (fifteen-entry single-scattering sets), native mesh, FP64 sums of a mixed-precision chain
        dict(name="fused_l3", kind="fused", struct="l3", rmax=5.4, legs=5, nk=0, fp64=False, absorbers=2),
        # the batched forward at scale: two absorbers of the packing, every path of up to 8 legs within 8 A, 401 k
        dict(name="fused_packing", kind="fused", struct="packing", rmax=8.0, legs=8, nk=401, fp64=False, absorbers=2),
        # the same in the plain FP64 form, a smaller cutoff
        dict(name="fused_packing_fp64", kind="fused", struct="packing", rmax=7.0, legs=7, nk=401, fp64=True, absorbers=2),
        # forward and backward (coordinates and per-path sigma^2) of one absorber's list
        dict(name="fused_packing_grad", kind="fused_grad", struct="packing", rmax=7.2, legs=7, nk=401, fp64=False,
             absorbers=1),
        # MD-EXAFS: thermal bcc Fe, 64 frames x 32 absorbers, every path of up to 3 legs within 5.5 A, mean per frame
        dict(name="md_bcc", kind="md", frames=64, absorbers=32, rmax=5.5, nk=0, fp64=False),
        # a reverse Monte Carlo step: rows of 32 absorbers of a NiO box, R-space misfit, gradient of every position
        dict(name="rmc_nio", kind="rmc", cells=8, absorbers=32, rmax=4.3, legs=4, nk=0, fp64=False),
        # the single scattering of a whole box from pair tables (every atom an absorber) and its gradient
        dict(name="pairs_nio", kind="pairs", cells=8, rmax=6.0, nk=0, fp64=False),
        # the path finder over MD frames (every absorber of every frame in one call)
        dict(name="finder_md", kind="finder", frames=16, absorbers=32, cells=8, rmax=5.5, legs=3, nk=0, fp64=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the listed kinds, sizes over their whole ranges."""
    kind = rng.choice(["dropin", "dropin_grad", "fused", "fused", "fused_grad", "fused_grad", "md", "rmc", "pairs",
                       "finder"])
    if kind in ("dropin", "dropin_grad"):
        legs = rng.randint(3, 5)
        return dict(kind=kind, struct=rng.choice(["cu", "packing"]), rmax=round(rng.uniform(4.2, 6.0), 2), legs=legs,
                    nk=rng.choice([0, 0, rng.randint(60, 401)]), fp64=rng.random() < 0.3,
                    take=int(_log(rng, 20, 4096 if kind == "dropin" else 2048)))
    if kind in ("fused", "fused_grad"):
        grad = kind == "fused_grad"
        rmax = round(rng.uniform(4.0, 6.5 if grad else 7.0), 2)
        return dict(kind=kind, struct=rng.choice(["packing", "packing", "l3"]), rmax=rmax, legs=rng.randint(3, 7),
                    nk=rng.choice([0, rng.randint(60, 401)]), fp64=rng.random() < 0.3, absorbers=rng.randint(1, 3))
    if kind == "md":
        return dict(kind=kind, frames=int(_log(rng, 1, 64)), absorbers=rng.randint(5, 32),
                    rmax=round(rng.uniform(4.5, 5.5), 2), nk=rng.choice([0, 0, rng.randint(60, 200)]),
                    fp64=rng.random() < 0.3)
    if kind == "rmc":
        return dict(kind=kind, cells=rng.randint(4, 8), absorbers=rng.randint(3, 40), rmax=round(rng.uniform(3.8, 4.6), 2),
                    legs=rng.randint(3, 4), nk=0, fp64=rng.random() < 0.3)
    if kind == "pairs":
        return dict(kind=kind, cells=rng.randint(4, 8), rmax=round(rng.uniform(4.5, 6.5), 2), nk=0, fp64=False)
    return dict(kind="finder", frames=int(_log(rng, 2, 24)), absorbers=rng.randint(2, 32), cells=rng.randint(5, 8),
                rmax=round(rng.uniform(4.0, 5.5), 2), legs=rng.randint(3, 4) if rng.random() < 0.3 else 3, nk=0, fp64=False)


# ------------------------------------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


_PHASES = {}


def _phase(struct, nk):
    """The structure's phase tables: native (nk 0) or resampled to nk points of the k range 0..20 1/A."""
    if (struct, nk) not in _PHASES:
        from feffgpu_b200.pad import phase_from_npz, resample_phase
        P = phase_from_npz(np.load(GOLDEN / (PHASE[struct] + ".npz"), allow_pickle=False), prefix="ph_")
        _PHASES[struct, nk] = resample_phase(P, np.linspace(0.0, 20.0, nk)) if nk else P
    return _PHASES[struct, nk]


def _q():
    return np.arange(NK) * 0.05


def _structure(struct, rmax, index):
    """Positions (n, 3) A of cluster `index` around an absorber at the origin (not included), and potentials (n,)."""
    rng = np.random.default_rng([index, 11])
    if struct == "cu":
        a, m = 3.61, 3
        g = np.array([[i, j, k] for i in range(-m, m + 1) for j in range(-m, m + 1) for k in range(-m, m + 1)], float)
        base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
        p = (g[:, None] + base[None]).reshape(-1, 3) * a
        r = np.linalg.norm(p, axis=1)
        p = p[(r > 1e-9) & (r < rmax + 0.5)]
        return p + rng.normal(0.0, 0.06, p.shape), np.ones(len(p), np.int64)
    # random sequential addition at the packing's density (0.08 1/A^3, no two atoms closer than 1.8 A)
    n = int(round(0.08 * 4.0 / 3.0 * math.pi * (rmax + 0.3) ** 3))
    pts = np.zeros((1, 3))
    while len(pts) <= n:
        c = rng.uniform(-(rmax + 0.3), rmax + 0.3, (64, 3))
        for x in c[np.linalg.norm(c, axis=1) < rmax + 0.3]:
            if len(pts) <= n and ((pts - x) ** 2).sum(1).min() > 1.8 ** 2:
                pts = np.concatenate([pts, x[None]])
    nph = int(_phase(struct, 0).nph)
    return pts[1:], rng.integers(1, nph + 1, len(pts) - 1)


def _enumerate(rel, rmax, legs):
    """Every path of 2..legs legs: {nleg: (sequences (B, nleg - 1) of indices into rel with len(rel) = the absorber,
    degeneracy (B,))}.  rel (n, 3): the candidates' positions relative to the absorber."""
    dev = rel.device
    n = rel.shape[0]
    pts = torch.cat([rel, torch.zeros(1, 3, device=dev, dtype=rel.dtype)])
    r = pts.norm(dim=1)
    D = torch.cdist(pts, pts)
    two_r = 2 * rmax
    seq = torch.nonzero(r[:n] <= rmax).to(torch.int64)
    length = r[seq[:, 0]]
    out = {2: (seq, torch.ones(len(seq), device=dev, dtype=torch.float64))}
    for m in range(1, legs - 1):
        last = seq[:, -1]
        new = length[:, None] + D[last]
        ok = (new + r[None, :] <= two_r) & (torch.arange(n + 1, device=dev)[None, :] != last[:, None])
        ok[:, :n] &= (r[:n] <= rmax)[None, :]
        par, j = torch.nonzero(ok, as_tuple=True)
        seq = torch.cat([seq[par], j[:, None]], 1)
        length = new[par, j]
        closed = seq[seq[:, -1] < n]
        rev = closed.flip(1)
        diff = (closed != rev).to(torch.int8)
        first = diff.argmax(1, keepdim=True)
        pal = diff.sum(1) == 0
        keep = pal | (closed.gather(1, first) < rev.gather(1, first))[:, 0]
        out[m + 2] = (closed[keep], torch.where(pal[keep], 1.0, 2.0).to(torch.float64))
    return out


def _paths(struct, rmax, legs, absorbers, seed):
    """[(coords (B, nleg, 3) FP64 (of FP32 values), ipots (B, nleg), deg (B,), row (B,))] over leg counts, on the
    device: the finder's list for `absorbers` clusters, row = absorber."""
    dev = _dev()
    per = {}
    for a in range(absorbers):
        p, ip = _structure(struct, rmax, a)
        rel = torch.tensor(p, device=dev, dtype=torch.float32)
        moved = p + np.random.default_rng([seed, a, 12]).normal(0.0, 0.03, p.shape)
        pts = torch.cat([torch.tensor(moved, device=dev, dtype=torch.float32), torch.zeros(1, 3, device=dev)])
        ips = torch.cat([torch.tensor(ip, device=dev), torch.zeros(1, device=dev, dtype=torch.int64)])
        for nleg, (seq, deg) in _enumerate(rel, rmax, legs).items():
            z = torch.full((len(seq), 1), len(rel), device=dev)
            full = torch.cat([z, seq], 1)
            per.setdefault(nleg, []).append((pts[full].double(), ips[full], deg,
                                             torch.full((len(seq),), a, device=dev, dtype=torch.int32)))
    return [tuple(torch.cat(x) for x in zip(*per[nleg])) for nleg in sorted(per)]


def _dropin_groups(case, seed):
    """The drop-in front end's chunks: `take` paths of the list, the longest leg count filled last."""
    groups = _paths(case["struct"], case["rmax"], case["legs"], 1, seed)
    left, out = case["take"], []
    for c, ip, deg, _row in groups:
        m = min(left, len(c))
        if m:
            # paths spread evenly over the leg count's list, in its order
            sel = (torch.arange(m, device=c.device) * len(c)) // m
            out.append((c[sel], ip[sel], deg[sel]))
            left -= m
    return out


def _md_groups(case, seed):
    """Thermal bcc Fe (a = 2.87 A, sigma 0.08 A): every 2- and 3-leg path of frames x absorbers clusters, the atoms
    moved on by the seed."""
    dev = _dev()
    a, rmax = 2.87, case["rmax"]
    g = np.arange(-5, 6)
    v = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    v = v[((v[:, 0] % 2) == (v[:, 1] % 2)) & ((v[:, 1] % 2) == (v[:, 2] % 2)) & (np.abs(v).sum(1) > 0)] * (a / 2)
    v = v[np.linalg.norm(v, axis=1) < rmax + 0.6]
    A = case["frames"] * case["absorbers"]
    def shifted(by, sigma, s):
        u = torch.randn(A, len(v) + 1, 3, device=dev, generator=torch.Generator(dev).manual_seed(s)) * sigma
        return by + u[:, 1:] - u[:, :1]

    rel = shifted(torch.tensor(v, device=dev, dtype=torch.float32)[None], 0.08, 3)
    now = shifted(rel, 0.03, seed + 4)
    r = rel.norm(dim=2)
    row = torch.arange(A, device=dev, dtype=torch.int32) // case["absorbers"]
    out = []
    s, i = torch.nonzero(r <= rmax, as_tuple=True)
    z3 = torch.zeros(len(s), 1, 3, device=dev)
    out.append((torch.cat([z3, now[s, i][:, None]], 1).double(), s, row[s]))
    parts = []
    for s0 in range(0, A, 512):
        rr, rl = r[s0:s0 + 512], rel[s0:s0 + 512]
        d = (rl[:, :, None] - rl[:, None]).norm(dim=3)
        ok = (rr[:, :, None] + d + rr[:, None, :] <= 2 * rmax) & (rr <= rmax)[:, :, None] & (rr <= rmax)[:, None, :]
        ok &= torch.ones_like(ok[0]).triu(1)
        s, i, j = torch.nonzero(ok, as_tuple=True)
        s = s + s0
        z3 = torch.zeros(len(s), 1, 3, device=dev)
        parts.append((torch.cat([z3, now[s, i][:, None], now[s, j][:, None]], 1).double(), s, row[s]))
    out.append(tuple(torch.cat(x) for x in zip(*parts)))
    groups = []
    for k, (c, s, rw) in enumerate(out):
        ip = torch.ones(len(c), c.shape[1], device=dev, dtype=torch.int64)
        ip[:, 0] = 0
        deg = torch.full((len(c),), (1.0 + (k > 0)) / case["absorbers"], device=dev, dtype=torch.float64)
        groups.append((c, ip, deg, rw))
    return groups


def _nio(cells, seed):
    """Disordered rock-salt NiO (a = 4.177 A, 5 % vacancies, sigma 0.1 A): positions, the positions moved by the seed,
    potentials (Ni 1, O 2), box."""
    a = 4.177
    g = np.array([[i, j, k] for i in range(cells) for j in range(cells) for k in range(cells)], float)
    fa = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    pos = np.concatenate([((g[:, None] + f[None]).reshape(-1, 3)) * a for f in (fa, fa + np.array([0.5, 0, 0]))])
    ip = np.repeat([1, 2], len(pos) // 2)
    rng = np.random.default_rng(5)
    keep = rng.random(len(pos)) >= 0.05
    pos = pos[keep] + rng.normal(0.0, 0.1, (int(keep.sum()), 3))
    return pos, pos + np.random.default_rng([seed, 5]).normal(0.0, 0.03, pos.shape), ip[keep], cells * a


def _rmc_inputs(case, seed):
    """(positions now, path groups as global atom indices, box) of a refinement step."""
    pos, now, ip, box = _nio(case["cells"], seed)
    rng = np.random.default_rng(6)
    ab = rng.choice(np.nonzero(ip == 1)[0], size=case["absorbers"], replace=False)
    x = torch.tensor(pos, device=_dev(), dtype=torch.float64)
    per = {}
    for a in ab:
        rel = x - x[a]
        rel = rel - box * torch.round(rel / box)
        near = torch.nonzero((rel.norm(dim=1) <= case["rmax"]) & (torch.arange(len(x), device=x.device) != int(a)))[:, 0]
        idx = torch.cat([near, torch.tensor([int(a)], device=x.device)])
        for nleg, (seq, deg) in _enumerate(rel[near], case["rmax"], case["legs"]).items():
            full = torch.cat([torch.full((len(seq), 1), len(near), device=x.device), seq], 1)
            at = idx[full]
            ipt = torch.tensor(ip, device=x.device)[at]
            ipt[at == int(a)] = 0
            per.setdefault(nleg, []).append((at, ipt, deg / len(ab)))
    groups = [tuple(torch.cat(v).cpu().numpy() for v in zip(*per[nleg])) for nleg in sorted(per)]
    return now, [g + (np.zeros(len(g[0]), int),) for g in groups], box


def _weights(seed, *shape):
    return torch.randn(*shape, device=_dev(), dtype=torch.float64, generator=torch.Generator(_dev()).manual_seed(seed + 17))


def _sigma2(seed, n):
    return 0.002 + 0.004 * torch.rand(n, device=_dev(), dtype=torch.float64,
                                      generator=torch.Generator(_dev()).manual_seed(seed + 29))


def _md_positions(case, seed):
    """(positions (F, n, 3) FP32, box, absorbers (F, A)) of thermal bcc Fe frames; the seed orders the frames and
    their absorbers."""
    n, a = case["cells"], 2.87
    g = np.array([[i, j, k] for i in range(n) for j in range(n) for k in range(n)], float)
    base = torch.tensor(np.concatenate([g, g + 0.5]) * a, device=_dev(), dtype=torch.float32)
    gen = torch.Generator(_dev()).manual_seed(41)
    pos = base[None] + 0.08 * torch.randn(case["frames"], len(base), 3, device=_dev(), generator=gen)
    rng = np.random.default_rng(8)
    ab = np.stack([rng.choice(len(base), size=case["absorbers"], replace=False) for _ in range(case["frames"])])
    rng = np.random.default_rng([seed, 8])
    order = rng.permutation(case["frames"])
    return pos[torch.tensor(order, device=pos.device)], n * a, rng.permuted(ab[order], axis=1)


# ------------------------------------------------------------------------------------------------ the user's program
def prepare(case, seed):
    from feffgpu_b200 import GPUPathStage, PathBatch
    kind = case["kind"]
    dtype = torch.complex128 if case["fp64"] else torch.complex64
    s = {"kind": kind}
    q = _q()
    if kind in ("dropin", "dropin_grad"):
        st = s["stage"] = GPUPathStage(_phase(case["struct"], case["nk"]), device="cuda", dtype=dtype)
        s["q"], s["S"] = q, st.linear_matrix(q)
        s["groups"] = [(c.to(st.rdtype), ip, deg.to(st.rdtype)) for c, ip, deg in _dropin_groups(case, seed)]
        if kind == "dropin_grad":
            s["w"] = _weights(seed, NK).to(st.rdtype)
    elif kind in ("fused", "fused_grad", "md"):
        struct = "bcc" if kind == "md" else case["struct"]
        groups = _md_groups(case, seed) if kind == "md" else _paths(struct, case["rmax"], case["legs"],
                                                                    case["absorbers"], seed)
        st = s["stage"] = GPUPathStage(_phase(struct, case["nk"]), device="cuda", dtype=dtype)
        s["batch"] = PathBatch(groups, nrows=case["frames"] if kind == "md" else case["absorbers"], device="cuda")
        s["q"], s["S"] = torch.tensor(q, device="cuda"), st.linear_matrix(q).double().contiguous()
        if kind == "fused_grad":
            s["coords"] = s["batch"].coords.clone().requires_grad_(True)
            s["sigma2"] = _sigma2(seed, s["batch"].n).requires_grad_(True)
            s["w"] = _weights(seed, s["batch"].nrows, NK)
    elif kind == "rmc":
        from feffgpu_b200.model import PathModel
        from feffgpu_b200.rspace import FitWindow, RSpaceMisfit
        pos, groups, box = _rmc_inputs(case, seed)
        st = GPUPathStage(_phase("nio", 0), device="cuda", dtype=dtype)
        m = s["model"] = PathModel(st, groups, pos, nrows=1, box=box)
        s["q"], s["S"] = torch.tensor(q, device="cuda"), st.linear_matrix(q).double().contiguous()
        target = _target(seed)
        s["misfit"] = RSpaceMisfit(NK, target, FitWindow(kmin=3.0, kmax=14.0, rmin=1.0, rmax=5.0), device="cuda")
        s["pos"] = torch.tensor(pos, device="cuda", dtype=torch.float64, requires_grad=True)
    elif kind == "pairs":
        from feffgpu_b200.pairs import PairTables
        _, pos, ip, box = _nio(case["cells"], seed)
        pt = s["tables"] = PairTables(_phase("nio", 0), q, box=box, rmax=case["rmax"], r_min=1.5, dr=0.002, device="cuda",
                                      dtype=dtype)
        pt.ipot = torch.tensor(ip)
        s["pos"] = torch.tensor(pos, device="cuda", dtype=torch.float64, requires_grad=True)
        s["w"] = _weights(seed, NK)
    else:
        from feffgpu_b200.pathfinder import GPUPathFinder
        s["finder"] = GPUPathFinder(_phase("bcc", 0), device="cuda", rmax=case["rmax"], nlegmax=case["legs"], critpw=0.0)
        s["pos"], s["box"], s["absorbers"] = _md_positions(case, seed)
        s["ipot"] = torch.ones(s["pos"].shape[1], device="cuda", dtype=torch.int64)
    return s


def _target(seed):
    """A measured spectrum on the fine grid: a few damped shells."""
    q = _q()
    rng = np.random.default_rng([seed, 9])
    chi = np.zeros(NK)
    for r, n, s2 in ((2.09, 6, 0.006), (2.95, 12, 0.007), (3.62, 8, 0.009), (4.18, 6, 0.01)):
        r = r + rng.normal(0.0, 0.01)
        chi += n / r ** 2 * np.exp(-2 * s2 * q ** 2 - 0.2 * r) * np.sin(2 * q * r + 0.3 * rng.normal()) / (1.0 + 0.3 * q)
    return chi


def run(s):
    kind = s["kind"]
    if kind in ("dropin", "dropin_grad"):
        st, rows, leaves = s["stage"], None, []
        for coords, ip, deg in s["groups"]:
            x = coords.requires_grad_(True) if kind == "dropin_grad" else coords
            leaves.append(x)
            cchi, reff = st.cchi(x, ip)
            chi = (st.chi_fine(cchi, reff, s["q"], s["S"]) * deg[:, None]).sum(0)
            rows = chi if rows is None else rows + chi
        if kind == "dropin":
            return rows
        return [rows.detach()] + list(torch.autograd.grad((rows * s["w"]).sum(), leaves))
    if kind in ("fused", "md"):
        with torch.no_grad():
            return s["stage"].chi_reduce(s["batch"], s["q"], s["S"])
    if kind == "fused_grad":
        rows = s["stage"].chi_reduce(s["batch"], s["q"], s["S"], coords=s["coords"], sigma2=s["sigma2"])
        return [rows.detach()] + list(torch.autograd.grad(rows, [s["coords"], s["sigma2"]], s["w"]))
    if kind == "rmc":
        rows = s["model"].rows(s["pos"], s["q"], s["S"])
        loss = s["misfit"](rows)[0]
        return [rows.detach(), loss.detach(), torch.autograd.grad(loss, s["pos"])[0]]
    if kind == "pairs":
        chi = s["tables"].single_scattering(s["pos"])
        return [chi.detach(), torch.autograd.grad((chi * s["w"]).sum(), s["pos"])[0]]
    res = s["finder"].enumerate_many(s["pos"], s["box"], s["absorbers"], s["ipot"])
    return [res["ref"]] + [t for nleg in sorted(res["paths"]) for t in res["paths"][nleg]]


# ------------------------------------------------------------------------------------------------ work
def _counts(case):
    """Expected paths per leg count, from the structure's density (no structure is built)."""
    kind, rmax = case["kind"], case["rmax"]
    if kind == "md":
        f = (rmax / 5.5) ** 3
        return {2: 58 * f * case["frames"] * case["absorbers"], 3: 205 * f * f * case["frames"] * case["absorbers"]}
    if kind == "rmc":
        f = (rmax / 4.2) ** 3
        c = {2: 28 * f, 3: 90 * f * f}
        if case["legs"] > 3:
            c[4] = 120 * f ** 3
        return {n: v * case["absorbers"] for n, v in c.items()}
    # the packing at 8 A: paths per absorber by leg count; the counts of seeded packings between 5 and 8 A follow the
    # cutoff to about the power 7 n - 13 (the shortest hop leaves long paths less room than their free atoms suggest)
    at8 = {2: 163, 3: 2200, 4: 17000, 5: 40000, 6: 30000, 7: 3600, 8: 8}
    out = {n: v * (rmax / 8.0) ** (3 if n == 2 else 7 * n - 13) * case.get("absorbers", 1) for n, v in at8.items()
           if n <= case["legs"]}
    if kind in ("dropin", "dropin_grad"):
        left, got = case["take"], {}
        for n in sorted(out):
            got[n] = min(left, out[n])
            left -= got[n]
        out = got
    return out


def work(case):
    kind = case["kind"]
    E = case["nk"] or 60
    if kind == "finder":
        A = case["frames"] * case["absorbers"]
        n = A * (263 if case["legs"] == 3 else 1500) * (case["rmax"] / 5.5) ** 6
        return {"bytes": n * (3 * 4 * 3 + 8 * 5 + 12) + case["frames"] * 2 * case["cells"] ** 3 * 12.0,
                "flops": n * 60 * 20.0}
    if kind == "pairs":
        atoms = 8 * case["cells"] ** 3 * 0.95
        pairs = atoms * 4.19 * case["rmax"] ** 3 * 0.104
        return {"bytes": atoms * 48.0 + 2 * 2 * ((case["rmax"] - 1.5) / 0.002) * NK * 8.0,
                "flops": atoms * atoms * 20.0 + pairs * 40.0}
    # operations of the reference's loops per (path, energy): affine in the partial waves per leg count (lmax 24)
    per = {2: 12342, 3: 17246, 4: 28718, 5: 40190, 6: 51662, 7: 63134, 8: 74606}
    cnt = _counts(case)
    flops = sum(v * per[n] * E for n, v in cnt.items())
    paths = sum(cnt.values())
    size = sum(v * n * (24 + 8) for n, v in cnt.items()) + paths * 20 + NK * 16.0
    if kind in ("fused_grad", "dropin_grad", "rmc"):
        flops *= 3
        size += sum(v * n * 24 for n, v in cnt.items()) + paths * 16
    return {"bytes": size, "flops": flops}


# ------------------------------------------------------------------------------------------------ exact
class _Tables:
    """The phase file's energy tables in complex128."""

    def __init__(self, P, dev):
        E = self.E = int(P.ne1)
        ph = np.asarray(P.ph)[:E, :, 0, :]
        lt, nph1 = int(P.ltot), int(P.nph) + 1
        em, eref = np.asarray(P.em)[:E], np.asarray(P.eref)[:E, 0]
        rkk = np.asarray(P.rkk)[:E, :, 0]
        e = em.real - float(P.edge)
        xk = np.sign(e) * np.sqrt(np.abs(2 * e))
        ck = np.sqrt(2 * (em - eref))
        lmax = np.zeros((nph1, E), np.int64)
        for ip in range(nph1):
            for ie in range(E):
                big = [l for l in range(int(P.lmax0[ip]), -1, -1) if abs(np.sin(ph[ie, l + lt, ip])) > 1e-7]
                lmax[ip, ie] = big[0] if big else 0
        L1 = self.L1 = int(lmax.max()) + 1
        t = np.zeros((nph1, L1 + 1, E), complex)
        for il in range(1, L1 + 1):
            l = il - 1
            tm, tp = ((np.exp(2j * ph[:, lt + s * l, :]) - 1) / 2j for s in (-1, 1))
            t[:, il] = (tm * (l + 1) + tp * l).T * (il <= lmax + 1)
        kinit = {1: -1, 4: -2}[int(P.ihole)]
        self.edge_l = 1 if kinit == -1 else 2
        wt = {}
        for k in (-1, 0, 1):
            kap = -kinit if k == 0 else kinit + k
            l = kap if kap > 0 else -kap - 1
            if l >= 0:
                wt[l] = wt.get(l, 0) - rkk[:, k + 1] ** 2 / (2 * l + 1) / 3
        c = lambda v: torch.tensor(v, device=dev)  # noqa: E731
        self.xk, self.ck, self.dk, self.lmax, self.t = c(xk), c(ck), c(ck - xk), c(lmax), c(t)
        self.wt = {l: c(v) for l, v in wt.items()}


def _lam(edge_l, ss):
    """(m, n) of the lambda set and the number of entries that reach the final state."""
    if not ss:
        return ([(0, 0), (-1, 0), (1, 0), (0, 1), (-2, 0), (2, 0)], 4) if edge_l == 1 else \
            ([(0, 0), (-1, 0), (1, 0), (-2, 0), (2, 0), (0, 1)], 6)
    out = []
    for n in range(edge_l + 1):
        for m in range(edge_l + 1):
            out += [(0, n)] if m == 0 else [(-m, n), (m, n)]
    return out, len(out)


def _xn(il, am):
    return math.sqrt((2 * il - 1) * math.factorial(il - 1 - am) / math.factorial(il - 1 + am)) if am < il else 0.0


def _wigner(beta, pairs, L1):
    """d^l_{m1 m2}(beta) for l = 0..L1 - 1 and the (m1, m2) of pairs, (L1, len(pairs), B): the explicit sum at
    l0 = max(|m1|, |m2|), then the three-term recursion."""
    f = math.factorial
    c2, s2, cb = torch.cos(beta / 2), torch.sin(beta / 2), torch.cos(beta)
    seeds = []
    for m1, m2 in pairs:
        l0, d = max(abs(m1), abs(m2)), 0
        for k in range(max(0, m2 - m1), min(l0 + m2, l0 - m1) + 1):
            w = math.sqrt(f(l0 + m1) * f(l0 - m1) * f(l0 + m2) * f(l0 - m2))
            w = w / (f(l0 + m2 - k) * f(k) * f(m1 - m2 + k) * f(l0 - m1 - k))
            d = d + (-1) ** (m1 - m2 + k) * w * c2 ** (2 * l0 + m2 - m1 - 2 * k) * s2 ** (m1 - m2 + 2 * k)
        seeds.append(d)
    seeds = torch.stack(seeds)
    l0 = torch.tensor([max(abs(m1), abs(m2)) for m1, m2 in pairs], device=beta.device)[:, None]
    mm = torch.tensor([m1 * m2 for m1, m2 in pairs], device=beta.device, dtype=torch.float64)[:, None]
    sq = torch.tensor([(m1 * m1, m2 * m2) for m1, m2 in pairs], device=beta.device, dtype=torch.float64)
    root = lambda l: torch.sqrt(((l * l - sq[:, 0]) * (l * l - sq[:, 1])).clamp(min=0.0))[:, None]  # noqa: E731
    out, prev, cur = [], torch.zeros_like(seeds), torch.zeros_like(seeds)
    for l in range(L1):
        if l:
            den = root(l) * max(l - 1, 1)
            nxt = ((2 * l - 1) * ((l - 1) * l * cb[None] - mm) * cur - l * root(l - 1) * prev) / den.clamp(min=1e-300)
            if l == 1:
                nxt = cb[None] * torch.ones_like(cur)                  # from d^0_00 = 1; the other pairs start later
            prev, cur = cur, torch.where(l > l0, nxt, torch.zeros_like(nxt))
        cur = torch.where(l0 == l, seeds, cur)
        out.append(cur)
    return torch.stack(out)


def _waves(z, L1, ncol):
    """c[il][j] for il = 1..L1 and columns j = 1..ncol, (L1, ncol, B, E)."""
    prev = torch.zeros((ncol,) + z.shape, device=z.device, dtype=z.dtype)
    prev[0] = 1.0
    cur, out = prev, [prev]
    for il in range(1, L1):
        prev, cur = cur, prev - (2 * il - 1) * z * (cur + torch.cat([torch.zeros_like(cur[:1]), cur[:-1]]))
        out.append(cur)
    return torch.stack(out)


def _geometry(x):
    """ri, beta, e^{-i eta} of legs 1..nleg from coordinates (B, nleg, 3) in bohr (FEFF's pathgeom)."""
    B, n, _ = x.shape
    at = [x[:, j % n] for j in range(n + 1)]
    ri, beta, al, ga = {}, {}, {}, {}

    def angles(v):
        r, rxy = v.norm(dim=1), torch.sqrt(v[:, 0] ** 2 + v[:, 1] ** 2)
        flat = rxy < 1e-6
        safe = torch.where(flat, torch.ones_like(rxy), rxy)
        ct, st = v[:, 2] / r, torch.where(flat, 0.0, rxy / r)
        return ct, st, torch.where(flat, torch.sign(ct), v[:, 0] / safe), torch.where(flat, 0.0, v[:, 1] / safe)

    def arg(re, im, other):
        re, im = (torch.where(v.abs() < 1e-6, torch.zeros_like(v), v) for v in (re, im))
        both = (re == 0) & (im == 0)
        return torch.where(both, other, torch.atan2(im, torch.where(both, torch.ones_like(re), re)))

    for j in range(1, n + 1):
        a, b, c = at[j], at[(j + 1) if j < n else 1], at[j - 1]
        ctp, stp, cpp, spp = angles(b - a)
        ct, st, cp, sp = angles(a - c)
        cppp, sppp = cp * cpp + sp * spp, spp * cp - cpp * sp
        phi, phip = torch.atan2(sp, cp), torch.atan2(spp, cpp)
        cosb = (ct * ctp + st * stp * cppp).clamp(-1.0, 1.0)
        u1, u2 = torch.stack([st * cp, st * sp, ct], 1), torch.stack([stp * cpp, stp * spp, ctp], 1)
        sinb = torch.sqrt((torch.linalg.cross(u1, u2) ** 2).sum(1) + 1e-30)
        a_j = arg(-(st * ctp - ct * stp * cppp), stp * sppp, phip - phi)
        g_j = arg(-(st * ctp * cppp - ct * stp), -st * sppp, torch.zeros_like(phi))
        al[j], ga[j], beta[j] = math.pi - g_j, math.pi - a_j, torch.atan2(sinb, cosb)
        ri[j] = (a - c).norm(dim=1)
    eta = {j: al[n if j == 1 else j - 1] + ga[j] for j in range(1, n + 1)}
    return ri, beta, {j: torch.polar(torch.ones_like(eta[j]), -eta[j]) for j in eta}


def _cchi(T, coords, ip):
    """cchi (B, E) complex128 and reff (B,) A of paths of one leg count."""
    B, n, _ = coords.shape
    ri, beta, ph = _geometry(coords / BOHR)
    lam, n0 = _lam(T.edge_l, n == 2)
    N, L1 = len(lam), T.L1
    ci, co = max(abs(m) + q + 1 for m, q in lam), max(q + 1 for _, q in lam)
    ip = torch.cat([ip, ip[:, :1]], 1)
    z = {j: -1j / (T.ck[None] * ri[j][:, None]) for j in ri}
    ent = [(i, j) for i in range(N) for j in range(N)]
    pairs = sorted({(lam[i][0], lam[j][0]) for i, j in ent})
    x = torch.tensor([[(-1) ** abs(m1) * _xn(il, abs(m1)) / _xn(il, abs(m2)) if abs(m1) < il and abs(m2) < il else 0.0
                       for m1, m2 in pairs] for il in range(1, L1 + 1)], device=coords.device, dtype=torch.float64)
    Q = None
    for k in range(1, n):
        win, wout = _waves(z[k + 1], L1, ci), _waves(z[k], L1, co)
        t = T.t[ip[:, k]][:, 1:].transpose(0, 1)                                          # (L1, B, E)
        D = (_wigner(beta[k], pairs, L1) * x[:, :, None]).permute(2, 1, 0)                # (B, pairs, L1)
        F = [None] * (N * N)
        for a in range(1, ci + 1):
            for b in range(1, co + 1):
                own = [q for q, (i, j) in enumerate(ent)
                       if abs(lam[i][0]) + lam[i][1] + 1 == a and lam[j][1] + 1 == b]
                if own:
                    X = torch.view_as_real((win[:, a - 1] * t * wout[:, b - 1]).transpose(0, 1).contiguous())
                    W = D[:, [pairs.index((lam[ent[q][0]][0], lam[ent[q][1]][0])) for q in own]]
                    R = torch.view_as_complex(torch.bmm(W, X.reshape(B, L1, -1)).reshape(B, len(own), T.E, 2).contiguous())
                    for r, q in enumerate(own):
                        F[q] = R[:, r]
        turn = torch.stack([ph[k + 1] ** m for m, _ in lam])
        F = torch.stack(F).reshape(N, N, B, T.E) * turn[:, None, :, None]
        Q = F[:, :n0] if Q is None else (F[:, :, None] * Q[None]).sum(1)
    la, l1, ln = (T.lmax[ip[:, j]] for j in (0, 1, n - 1))
    lx1, lxn = torch.maximum(la, l1) + 1, torch.maximum(ln, la) + 1
    it = T.edge_l + 1
    c1, cn = _waves(z[1], it, ci), _waves(z[n], it, co)
    dn = _wigner(beta[n], pairs, it)

    def keep(v, il, col, lx):          # the stage's truncation of a leg's partial waves
        return v[il - 1, col - 1] if col == 1 and il <= 2 else torch.where(il <= lx, v[il - 1, col - 1], 0.0)

    ptrac = 0
    for l, W in T.wt.items():
        il = l + 1
        s = 0
        for a in range(n0):
            m, q = lam[a]
            if abs(m) + 1 > il or abs(m) + q + 1 > il:
                continue
            g1 = keep(c1, il, abs(m) + q + 1, lx1) * ((-1) ** abs(m) * _xn(il, abs(m))) * (ph[1] ** m)[:, None]
            x = 0
            for b in range(n0):
                mb, qb = lam[b]
                if abs(mb) + 1 > il:
                    continue
                g2 = keep(cn, il, qb + 1, lxn) * ((2 * il - 1) / _xn(il, abs(mb)))
                x = x + g2 * dn[l, pairs.index((m, mb))][:, None] * Q[b, a]
            s = s + g1 * x
        ptrac = ptrac + W[None] * s
    reff = sum(ri.values()) / 2
    rho = 1
    for j in ri:
        rho = rho * (T.ck[None] * ri[j][:, None])
    out = ptrac * torch.exp(2j * reff[:, None] * T.dk[None]) / rho
    return torch.where(T.ck.abs()[None] <= 1e-16, torch.zeros_like(out), out), reff * BOHR


def _chi(T, coords, ip, q, sigma2=None):
    """chi (B, NK) of paths: amplitude and unwrapped phase interpolated linearly in k, damped."""
    c, reff = _cchi(T, coords, ip)
    amp = torch.sqrt(c.real ** 2 + c.imag ** 2 + 1e-30)
    live = amp >= 1e-16
    ang = torch.where(live, torch.atan2(torch.where(live, c.imag, 0.0), torch.where(live, c.real, 1.0)), 0.0)
    d = torch.diff(ang, dim=1)
    d = d - 2 * math.pi * torch.round((d / (2 * math.pi)).detach())
    pha = torch.cat([ang[:, :1], ang[:, :1] + torch.cumsum(d, 1)], 1)
    kf = T.xk / BOHR
    qc = q.clamp(float(kf[0]), float(kf[-1]))
    j = (torch.searchsorted(kf, qc, right=True) - 1).clamp(0, T.E - 2)
    f = (qc - kf[j]) / (kf[j + 1] - kf[j])
    a, p = (v[:, j] * (1 - f) + v[:, j + 1] * f for v in (amp, pha))
    out = a * torch.sin(p + 2 * q[None] * reff[:, None])
    return out if sigma2 is None else out * torch.exp(-2 * sigma2[:, None] * q[None] ** 2)


def _rows(T, groups, nrows, q, chunk, grad=None):
    """rows (nrows, NK) of groups (coords, ipots, deg, row[, sigma2]); with grad (nrows, NK) also the gradients of
    (rows * grad).sum() per group: [(dcoords, dsigma2 or None)]."""
    rows = torch.zeros(nrows, len(q), device=q.device, dtype=torch.float64)
    grads = []
    for g in groups:
        c, ip, deg, row = g[:4]
        s2 = g[4] if len(g) > 4 else None
        dc, ds = torch.zeros_like(c), None if s2 is None else torch.zeros_like(s2)
        for i in range(0, len(c), chunk):
            sl = slice(i, i + chunk)
            if grad is None:
                with torch.no_grad():
                    v = _chi(T, c[sl], ip[sl], q, None if s2 is None else s2[sl]) * deg[sl, None]
            else:
                x = c[sl].detach().clone().requires_grad_(True)
                y = None if s2 is None else s2[sl].detach().clone().requires_grad_(True)
                v = _chi(T, x, ip[sl], q, y) * deg[sl, None]
                got = torch.autograd.grad((v * grad[row[sl].long()]).sum(), [x] + ([] if y is None else [y]))
                dc[sl] = got[0]
                if y is not None:
                    ds[sl] = got[1]
            rows.index_add_(0, row[sl].long(), v.detach())
        grads.append((dc, ds))
    return rows, grads


def exact(case, seed):
    kind, dev = case["kind"], _dev()
    q = torch.tensor(_q(), device=dev)
    if kind == "finder":
        return None
    struct = {"md": "bcc", "rmc": "nio", "pairs": "nio"}.get(kind) or case["struct"]
    T = _Tables(_phase(struct, case["nk"]), dev)
    chunk = 4096 * 401 // T.E            # paths at a time
    back = chunk // (16 if struct == "l3" else 8)
    if kind in ("dropin", "dropin_grad"):
        real = torch.float64 if case["fp64"] else torch.float32
        groups = [(c.to(real).double(), ip, deg, torch.zeros(len(c), device=dev))
                  for c, ip, deg in _dropin_groups(case, seed)]
        if kind == "dropin":
            return _rows(T, groups, 1, q, chunk)[0][0]
        rows, grads = _rows(T, groups, 1, q, back, _weights(seed, 1, NK).to(real).double())
        return [rows[0]] + [g for g, _ in grads]
    if kind in ("fused", "md"):
        groups = _md_groups(case, seed) if kind == "md" else _paths(struct, case["rmax"], case["legs"],
                                                                    case["absorbers"], seed)
        return _rows(T, groups, case["frames"] if kind == "md" else case["absorbers"], q, chunk)[0]
    if kind == "fused_grad":
        groups = _paths(struct, case["rmax"], case["legs"], case["absorbers"], seed)
        s2 = _split(_sigma2(seed, sum(len(g[0]) for g in groups)), groups)
        rows, grads = _rows(T, [g + (v,) for g, v in zip(groups, s2)], case["absorbers"], q, back,
                            _weights(seed, case["absorbers"], NK))
        n = max(g[0].shape[1] for g in groups)
        pad = [torch.nn.functional.pad(dc, (0, 0, 0, n - dc.shape[1])) for dc, _ in grads]
        return [rows, torch.cat(pad), torch.cat([ds for _, ds in grads])]
    if kind == "rmc":
        pos, groups, box = _rmc_inputs(case, seed)
        x = torch.tensor(pos, device=dev, requires_grad=True)
        lst = []
        for at, ip, deg, row in groups:
            at = torch.tensor(at, device=dev)
            rel = x[at] - x[at[:, :1]]
            lst.append((rel - box * torch.round((rel / box).detach()), torch.tensor(ip, device=dev),
                        torch.tensor(deg, device=dev), torch.tensor(row, device=dev)))
        det = [(v[0].detach(),) + v[1:] for v in lst]
        rows, _ = _rows(T, det, 1, q, chunk)
        chi = rows[0].clone().requires_grad_(True)
        F = _transform(dev)
        t = F @ torch.tensor(_target(seed), device=dev).to(torch.complex128)
        loss = ((F @ chi.to(torch.complex128) - t).abs() ** 2).sum() / (t.abs() ** 2).sum()
        (g,) = torch.autograd.grad(loss, chi)
        _, grads = _rows(T, det, 1, q, back, g[None])
        total = sum((c * dc).sum() for (c, *_), (dc, _s) in zip(lst, grads))
        return [rows, loss.detach(), torch.autograd.grad(total, x)[0]]
    # pair tables: the two-leg tables on the distance grid, linear interpolation between grid points
    _, pos, ip, box = _nio(case["cells"], seed)
    r0, dr = 1.5, 0.002
    nr = int(round((case["rmax"] - r0) / dr)) + 1
    tabs = []
    for p in (1, 2):
        c = torch.zeros(nr, 2, 3, device=dev, dtype=torch.float64)
        c[:, 1, 2] = r0 + dr * torch.arange(nr, device=dev, dtype=torch.float64)
        with torch.no_grad():
            tabs.append(_chi(T, c, torch.tensor([[0, p]], device=dev).repeat(nr, 1), q))
    Tb = torch.stack(tabs)
    w, x, ipt = _weights(seed, NK), torch.tensor(pos, device=dev), torch.tensor(ip, device=dev)
    D, n = Tb @ w, len(pos)
    hist, grad = torch.zeros(2 * nr, device=dev, dtype=torch.float64), torch.zeros_like(x)
    for i in range(0, n, 512):
        rel = x[None] - x[i:i + 512, None]
        rel = rel - box * torch.round(rel / box)
        r2 = (rel ** 2).sum(2)
        a, j = torch.nonzero((r2 <= case["rmax"] ** 2) & (r2 > 1e-6), as_tuple=True)
        rel, r, p = rel[a, j], r2[a, j].sqrt(), ipt[j] - 1
        u = (r - r0) / dr
        i0 = u.floor().clamp(0, nr - 2)
        f = (u - i0).clamp(0.0, 1.0)
        at = p * nr + i0.long()
        hist.index_add_(0, at, 1 - f)
        hist.index_add_(0, at + 1, f)
        slope = torch.where((u - i0 >= 0) & (u - i0 <= 1), (D.reshape(-1)[at + 1] - D.reshape(-1)[at]) / dr, 0.0) / n
        gv = (slope / r)[:, None] * rel
        grad.index_add_(0, j, gv)
        grad.index_add_(0, a + i, -gv)
    return [hist @ Tb.reshape(2 * nr, -1) / n, grad]


def _split(v, groups):
    return list(torch.split(v, [len(g[0]) for g in groups]))


def _transform(dev):
    """The R-space transform of the refinement's window (k 3-14, Hanning sills 1 wide, k^2; R 1-5 A), (NR, NK)."""
    k, nfft = 0.05 * np.arange(NK), 2048
    rise = 0.5 * (1 - np.cos(np.pi * np.clip(k - 2.5, 0, 1)))
    fall = 0.5 * (1 + np.cos(np.pi * np.clip(k - 13.5, 0, 1)))
    r = np.float32(math.pi / (0.05 * nfft)) * np.arange(nfft // 2, dtype=np.float32)
    m = np.nonzero((r >= np.float32(1.0)) & (r <= np.float32(5.0)))[0]
    F = np.exp(-2j * np.pi * np.outer(m, np.arange(NK)) / nfft) * (0.05 / math.sqrt(math.pi)) * (rise * fall * k ** 2)[None]
    return torch.tensor(F, device=dev)
