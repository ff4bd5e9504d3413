"""Workloads of the framework, one pass each through its public entry points.

A case names the stage it runs (``kind``) and that stage's sizes and options:

* ``rms``      Context.knn_rms: trajectory frames against themselves or against
               a separate reference set, host (numpy) or device frames, sorted
               neighbour lists or full distance rows;
* ``vec``      Context.knn_data: feature vectors (sin/cos of dihedral angles);
* ``contact``  Context.contact_profile, then Context.knn_data_sparse on the
               contact maps it returns;
* ``graph``    Context.sysparse / Context.gesparse on neighbour lists;
* ``eig``      Context.decomp_sparse and its variants (a sigma per landmark,
               Nystrom extension of out-of-sample queries);
* ``serve``    a resident Server answering query requests.

Inputs are synthetic and made from the seed alone: trajectories are a chain
with 0.15 nm bonds in metastable basins with Ornstein-Uhlenbeck drift per atom,
rotated and translated rigidly per frame and rounded to the 0.001 nm of the XTC
format; vectors come from a mixture of wrapped normals; graphs from points on a
rolled strip.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from mdsctk_gb300 import Context
from mdsctk_gb300.serve import Server


def listed():
    return [
        # a short peptide trajectory clustered from a script with the defaults: numpy arrays in and out; launches and copies count
        {"name": "peptide_host", "kind": "rms", "n_ref": 1000, "n_fit": 0, "atoms": 60, "k": 20, "precision": "fp32", "host": True, "nofit": False, "full": False},
        # the benchmark's own workload: all pairs of a protein trajectory, frames already on the device
        {"name": "protein_20k", "kind": "rms", "n_ref": 20000, "n_fit": 0, "atoms": 1000, "k": 100, "precision": "bf16x3", "host": False, "nofit": False, "full": False},
        # the largest all-pairs run: a long backbone trajectory
        {"name": "backbone_100k", "kind": "rms", "n_ref": 100000, "n_fit": 0, "atoms": 304, "k": 64, "precision": "bf16x3", "host": False, "nofit": False, "full": False},
        # out-of-sample frames against landmarks, as the tool reads them from files: host arrays, sizes that fill no tile
        {"name": "queries_host", "kind": "rms", "n_ref": 20011, "n_fit": 2047, "atoms": 304, "k": 50, "precision": "bf16x3", "host": True, "nofit": False, "full": False},
        # the unsorted full distance matrix (-s false), input of dense methods
        {"name": "full_rows", "kind": "rms", "n_ref": 3001, "n_fit": 0, "atoms": 257, "k": 0, "precision": "fp32", "host": False, "nofit": False, "full": True},
        # the vector benchmark: dihedral features of a long trajectory
        {"name": "vectors_200k", "kind": "vec", "n_ref": 200000, "n_fit": 0, "dim": 64, "k": 32, "correlation": False, "precision": "bf16x3", "host": False},
        # correlation distance of new vectors to a reference set, default options, host arrays, odd sizes
        {"name": "correlation_host", "kind": "vec", "n_ref": 20011, "n_fit": 5003, "dim": 50, "k": 20, "correlation": True, "precision": "fp32", "host": True},
        # contact maps of a trajectory and their nearest neighbours
        {"name": "contacts", "kind": "contact", "frames": 8000, "atoms": 304, "eps": 12.0, "k": 32},
        # the sparse neighbour matrix of a long trajectory's lists
        {"name": "graph_100k", "kind": "graph", "n": 100000, "k": 64, "mode": "sys"},
        # the spectral embedding of a small data set with the reference's default Krylov size
        {"name": "spectral_2k", "kind": "eig", "n": 2000, "m": 0, "k": 50, "nev": 10, "auto": False},
        # landmarks with a sigma each, and the Nystrom extension of many more queries than landmarks
        {"name": "nystrom_auto_20k", "kind": "eig", "n": 20001, "m": 50003, "k": 30, "nev": 10, "auto": True},
        # a serving process: requests of one frame, some frames and many frames that arrive together
        {"name": "serving", "kind": "serve", "n": 20000, "atoms": 304, "k": 50, "nev": 10, "requests": "1,33,500"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rms", "rms", "vec", "contact", "graph", "eig", "serve"])
    if kind == "rms":
        full = rng.random() < 0.15
        atoms = _log_int(rng, 40, 1200)
        # no more pair work than the largest listed run
        top = min(4000 if full else 60000, int(math.sqrt(8.0e12 / 18 / atoms)))
        n_ref = _log_int(rng, 500, top)
        n_fit = _log_int(rng, 100, n_ref) if rng.random() < 0.4 else 0
        tc = rng.random() < 0.6 or n_ref > 12000
        return {"kind": "rms", "n_ref": n_ref, "n_fit": n_fit, "atoms": atoms, "k": 0 if full else _log_int(rng, 8, 120),
                "precision": "bf16x3" if tc else "fp32", "host": rng.random() < 0.5, "nofit": rng.random() < 0.15, "full": full}
    if kind == "vec":
        n_ref = _log_int(rng, 1000, 150000)
        n_fit = _log_int(rng, 500, n_ref) if rng.random() < 0.4 else 0
        tc = rng.random() < 0.6 or n_ref > 30000
        return {"kind": "vec", "n_ref": n_ref, "n_fit": n_fit, "dim": _log_int(rng, 8, 120), "k": _log_int(rng, 5, 60),
                "correlation": rng.random() < 0.35, "precision": "bf16x3" if tc else "fp32", "host": rng.random() < 0.5}
    if kind == "contact":
        return {"kind": "contact", "frames": _log_int(rng, 500, 8000), "atoms": _log_int(rng, 60, 304), "eps": round(rng.uniform(7.0, 13.0), 2), "k": _log_int(rng, 8, 64)}
    if kind == "graph":
        return {"kind": "graph", "n": _log_int(rng, 1000, 100000), "k": _log_int(rng, 8, 64), "mode": rng.choice(["sys", "sys", "ge", "ge_sym"])}
    if kind == "eig":
        n = _log_int(rng, 800, 20000)
        return {"kind": "eig", "n": n, "m": _log_int(rng, 500, 50000) if rng.random() < 0.5 else 0, "k": rng.randint(20, 50), "nev": rng.randint(4, 10), "auto": rng.random() < 0.5}
    requests = ",".join(str(_log_int(rng, 1, 500)) for _ in range(rng.randint(1, 4)))
    return {"kind": "serve", "n": _log_int(rng, 2000, 20000), "atoms": _log_int(rng, 60, 304), "k": rng.randint(20, 60), "nev": rng.randint(4, 10), "requests": requests}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _context():
    return Context(0)  # a program keeps one


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _trajectory(n, atoms, g, basins=8, sigma=0.08, tau=200.0, dwell=500.0):
    """[n, atoms, 3] float32 nm on the GPU."""
    dev = "cuda"
    step = torch.randn(atoms, 3, generator=g, device=dev)
    chain = torch.cumsum(0.15 * step / step.norm(dim=1, keepdim=True), 0)
    chain = chain - chain.mean(0)
    # basins: smooth displacement fields along the chain, a dwell time per visit
    t = torch.linspace(0, 1, atoms, device=dev)[:, None]
    fields = torch.zeros(basins, atoms, 3, device=dev)
    for h in range(1, 7):
        phase = 2 * math.pi * torch.rand(basins, 1, 1, generator=g, device=dev)
        fields += torch.sin(h * math.pi * t + phase) * (0.25 * torch.randn(basins, 1, 3, generator=g, device=dev))
    switch = torch.rand(n, generator=g, device=dev) < 1.0 / dwell
    visits = torch.cumsum(switch.to(torch.int64), 0)
    state = torch.randint(basins, (n + 1,), generator=g, device=dev)[visits]
    # Ornstein-Uhlenbeck drift, a block of frames at a time
    a = math.exp(-1.0 / tau)
    block = 128
    i = torch.arange(block, device=dev)
    lag = (i[:, None] - i[None, :]).clamp(min=0).to(torch.float32)
    mix = torch.tril(a ** lag) * (sigma * math.sqrt(1 - a * a))
    decay = (a ** (i + 1).to(torch.float32))[:, None]
    x = torch.empty(n, atoms * 3, device=dev)
    last = sigma * torch.randn(1, atoms * 3, generator=g, device=dev)
    for f in range(0, n, block):
        m = min(block, n - f)
        noise = torch.randn(m, atoms * 3, generator=g, device=dev)
        x[f:f + m] = mix[:m, :m] @ noise + decay[:m] * last
        last = x[f + m - 1:f + m]
    x = x.view(n, atoms, 3)
    for f in range(0, n, 8192):
        part = x[f:f + 8192]
        part += chain + fields[state[f:f + 8192]]
        q = torch.randn(part.shape[0], 4, generator=g, device=dev)
        w, u, v, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
        rot = torch.stack([1 - 2 * (v * v + z * z), 2 * (u * v - w * z), 2 * (u * z + w * v),
                           2 * (u * v + w * z), 1 - 2 * (u * u + z * z), 2 * (v * z - w * u),
                           2 * (u * z - w * v), 2 * (v * z + w * u), 1 - 2 * (u * u + v * v)], 1).view(-1, 3, 3)
        moved = torch.einsum("fij,faj->fai", rot, part) + 5 * torch.rand(part.shape[0], 1, 3, generator=g, device=dev)
        x[f:f + 8192] = torch.round(moved * 1000.0) / 1000.0
    return x


def _vectors(n, dim, g, components=12):
    dev = "cuda"
    angles = (dim + 1) // 2
    centre = (2 * torch.rand(components, angles, generator=g, device=dev) - 1) * math.pi
    width = (2 + 18 * torch.rand(components, angles, generator=g, device=dev)) ** -0.5
    weight = torch.rand(components, generator=g, device=dev) + 0.1
    edge = torch.cumsum(weight / weight.sum(), 0)
    comp = torch.searchsorted(edge, torch.rand(n, generator=g, device=dev)).clamp(max=components - 1)
    ang = centre[comp] + width[comp] * torch.randn(n, angles, generator=g, device=dev)
    out = torch.stack([torch.sin(ang), torch.cos(ang)], 2).view(n, 2 * angles)[:, :dim]
    return out.to(torch.float64).contiguous()


def _lists(n, k, g):
    """Neighbour lists of frames along a random walk, in shuffled order: distances [n, k] f64 ascending, indices [n, k] i32.
    The walk is the same for every seed, its scale and the order of the frames are the seed's: so every seed's matrix has as many entries."""
    dev = "cuda"
    p = torch.cumsum(torch.randn(n, 3, generator=_generator(n * 1000 + k), device=dev, dtype=torch.float64), 0)
    p = p * (0.5 + torch.rand(1, generator=g, device=dev, dtype=torch.float64))
    near = torch.cat([torch.arange(-k, 0, device=dev), torch.arange(1, k + 1, device=dev)])
    label = torch.randperm(n, generator=g, device=dev)
    dist = torch.empty(n, k, dtype=torch.float64, device=dev)
    idx = torch.empty(n, k, dtype=torch.int32, device=dev)
    for r in range(0, n, 16384):
        row = torch.arange(r, min(r + 16384, n), device=dev)
        col = row[:, None] + near[None, :]
        inside = (col >= 0) & (col < n)
        col = col.clamp(0, n - 1)
        d = (p[row][:, None, :] - p[col]).square().sum(2).sqrt().masked_fill(~inside, math.inf)
        v, o = torch.sort(d, dim=1, stable=True)
        dist[label[row]] = v[:, :k]
        idx[label[row]] = label[torch.gather(col, 1, o[:, :k])].to(torch.int32)
    return dist, idx


def _strip(n, g):
    """Points on a rolled strip (swiss roll)."""
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    v = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    t = 1.5 * math.pi * (1 + 2 * u)
    return torch.stack([t * torch.cos(t), 21 * v, t * torch.sin(t)], 1)


def _near(x, y, k, same):
    """The k nearest points y of each point x: distances and indices."""
    dist, idx = [], []
    for r in range(0, x.shape[0], 1024):
        q = x[r:r + 1024]
        d2 = torch.zeros(q.shape[0], y.shape[0], dtype=torch.float64, device="cuda")
        for c in range(3):
            d2 += (q[:, c, None] - y[None, :, c]).square()
        if same:
            i = torch.arange(q.shape[0], device="cuda")
            d2[i, i + r] = math.inf
        v, o = torch.topk(d2, k, dim=1, largest=False)
        dist.append(v.sqrt())
        idx.append(o)
    return torch.cat(dist), torch.cat(idx)


def _requests(case):
    return [int(v) for v in case["requests"].split(",")]


def prepare(case, seed):
    g = _generator(seed)
    s = {"case": case}
    kind = case["kind"]
    if kind == "rms":
        x = _trajectory(case["n_ref"] + case["n_fit"], case["atoms"], g)
        mass = torch.tensor([12.011, 14.007, 15.999, 12.011], device="cuda").repeat(case["atoms"] // 4 + 1)[:case["atoms"]].contiguous()
        ref, fit = x[:case["n_ref"]], (x[case["n_ref"]:] if case["n_fit"] else None)
        if case["host"]:
            s.update(ref=ref.cpu().numpy(), fit=None if fit is None else fit.cpu().numpy(), mass=mass.cpu().numpy())
        else:
            s.update(ref=ref.contiguous(), fit=None if fit is None else fit.contiguous(), mass=mass)
    elif kind == "vec":
        x = _vectors(case["n_ref"] + case["n_fit"], case["dim"], g)
        ref, fit = x[:case["n_ref"]], (x[case["n_ref"]:] if case["n_fit"] else None)
        if case["host"]:
            s.update(ref=ref.cpu().numpy(), fit=None if fit is None else fit.cpu().numpy())
        else:
            s.update(ref=ref.contiguous(), fit=None if fit is None else fit.contiguous())
    elif kind == "contact":
        half = case["atoms"] // 2
        # (one trajectory for every seed, which sets the frame it starts at and its direction in time, so that every seed has as many contacts)
        x = _trajectory(case["frames"], case["atoms"], _generator(case["frames"] * 1000 + case["atoms"]))
        at, back = torch.randint(case["frames"], (2,), generator=g, device="cuda").tolist()
        x = torch.roll(x, at, 0)
        x = x.flip(0) if back % 2 else x
        # the maps' values, all 1.0, which the tools keep in a file beside the indices
        total = sum(int((torch.cdist(p[:, :half], p[:, half:]) * 10 < case["eps"]).sum()) for p in torch.split(x, 512))
        s.update(xyz=x.cpu().numpy(), g1=np.arange(0, half, dtype=np.int32), g2=np.arange(half, case["atoms"], dtype=np.int32),
                 ones=np.ones(total + total // 64 + 4096))
    elif kind == "graph":
        dist, idx = _lists(case["n"], case["k"], g)
        s.update(dist=dist.cpu().numpy(), idx=idx.cpu().numpy())
    elif kind == "eig":
        n, k = case["n"], case["k"]
        pts = _strip(n + case["m"], g)
        land = pts[:n]
        dist, idx = _near(land, land, k, True)
        row = torch.arange(n, device="cuda")[:, None].expand(n, k)
        key = torch.unique(torch.minimum(row, idx) * n + torch.maximum(row, idx))
        col, low = key // n, key % n
        d = (land[col] - land[low]).square().sum(1).sqrt()
        pcol = torch.searchsorted(col, torch.arange(n + 1, device="cuda"))
        s.update(pcol=pcol.to(torch.int32).cpu().numpy(), irow=low.to(torch.int32).cpu().numpy(), dist=d.cpu().numpy(), sigma=float(dist.median()))
        if case["m"]:
            qd, qi = _near(pts[n:], land, k, False)
            o = torch.argsort(qi, dim=1)
            s.update(pcolB=np.arange(case["m"] + 1, dtype=np.int32) * np.int32(k), irowB=torch.gather(qi, 1, o).to(torch.int32).reshape(-1).cpu().numpy(),
                     distB=torch.gather(qd, 1, o).reshape(-1).cpu().numpy())
        # eigenvectors are compared up to sign: each is turned to have a positive product with this vector
        s["probe"] = torch.randn(n, generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    elif kind == "serve":
        sizes = _requests(case)
        x = _trajectory(case["n"] + sum(sizes), case["atoms"], g).cpu().numpy()
        cut = np.cumsum([case["n"]] + sizes)
        s["queries"] = [np.ascontiguousarray(x[a:b]) for a, b in zip(cut[:-1], cut[1:])]
        s["server"] = Server(x[:case["n"]], k=case["k"], sigma=1.0, nev=case["nev"], max_batch_frames=1024, slots=2, hbm_budget=8 << 30)
    return s


# -------------------------------------------------------------------- passes
def _signed(probe, vectors, *others):
    turn = np.where(vectors @ probe < 0, -1.0, 1.0)[:, None]
    return [v * turn for v in (vectors,) + others]


def run(s):
    c, kind = s["case"], s["case"]["kind"]
    if kind == "rms":
        d, i = _context().knn_rms(s["ref"], s["fit"], s["mass"], c["k"], nofit=c["nofit"], sort=not c["full"], precision=c["precision"])
        return {"d": d, "i": i}
    if kind == "vec":
        d, i = _context().knn_data(s["ref"], s["fit"], c["k"], correlation=c["correlation"], precision=c["precision"])
        return {"d": d, "i": i}
    if kind == "contact":
        off, idx = _context().contact_profile(s["xyz"], s["g1"], s["g2"], c["eps"])
        d, i = _context().knn_data_sparse((off, idx, s["ones"][:len(idx)]), None, c["k"])
        return {"off": off, "idx": idx, "d": d, "i": i}
    if kind == "graph":
        if c["mode"] == "sys":
            _, pcol, irow, val = _context().sysparse(s["dist"], s["idx"])
        else:
            _, pcol, irow, val = _context().gesparse(s["dist"], s["idx"], symmetric=c["mode"] == "ge_sym")
        return {"pcol": pcol, "irow": irow, "val": val}
    if kind == "eig":
        # (the residuals, which are rounding noise once a pair has converged, are not returned)
        a, n, nev, k_sigma = (s["pcol"], s["irow"], s["dist"]), c["n"], c["nev"], c["k"] // 4
        if c["m"]:
            b = (c["m"], s["pcolB"], s["irowB"], s["distB"])
            if c["auto"]:
                w, v, ext, _, nconv, sig = _context().auto_decomp_sparse_nystrom(n, *a, *b, k_sigma, nev)
            else:
                w, v, ext, _, nconv = _context().decomp_sparse_nystrom(n, *a, *b, s["sigma"], nev)
            v, ext = _signed(s["probe"], v, ext)
        else:
            if c["auto"]:
                w, v, _, nconv, sig = _context().auto_decomp_sparse(n, *a, k_sigma, nev)
            else:
                w, v, _, nconv = _context().decomp_sparse(n, *a, s["sigma"], nev)
            v, = _signed(s["probe"], v)
        out = {"evals": w, "evecs": v, "nconv": nconv}
        if c["m"]:
            out["ext"] = ext
        if c["auto"]:
            out["sigmas"] = sig
        return out
    tickets = [s["server"].submit(q) for q in s["queries"]]
    answers = [s["server"].wait(t) for t in tickets]
    return [{"ext": ext, "d": d, "i": i} for ext, d, i, _ in answers]


# ---------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; the arithmetic of the pairs that are reported (a full matrix reports every pair), and of a Krylov space for the eigenpairs."""
    kind = case["kind"]
    if kind == "rms":
        n_fit = case["n_fit"] or case["n_ref"]
        width = case["n_ref"] if case["full"] else case["k"]
        frames = case["n_ref"] + case["n_fit"]
        return {"bytes": 12.0 * case["atoms"] * frames + 12.0 * n_fit * width, "flops": 18.0 * case["atoms"] * n_fit * (width + (0 if case["full"] else 1))}
    if kind == "vec":
        n_fit = case["n_fit"] or case["n_ref"]
        return {"bytes": 8.0 * case["dim"] * (case["n_ref"] + case["n_fit"]) + 12.0 * n_fit * case["k"], "flops": 3.0 * case["dim"] * n_fit * (case["k"] + 1)}
    if kind == "contact":
        pairs = (case["atoms"] // 2) * (case["atoms"] - case["atoms"] // 2)
        return {"bytes": 12.0 * case["atoms"] * case["frames"] + 12.0 * case["frames"] * case["k"], "flops": 8.0 * pairs * case["frames"]}
    if kind == "graph":
        return {"bytes": (12.0 + 8.0) * case["n"] * case["k"], "flops": 0.0}
    if kind == "eig":
        n, k, nev = case["n"], case["k"], case["nev"]
        nnz, ncv = 0.6 * n * k, min(10 * nev + 1, n)
        return {"bytes": 12.0 * nnz + 8.0 * n * nev + case["m"] * (12.0 * k + 8.0 * nev), "flops": 4.0 * nnz * ncv + 2.0 * n * ncv * ncv + 2.0 * case["m"] * k * nev}
    m = sum(_requests(case))
    return {"bytes": 12.0 * case["atoms"] * (case["n"] + m) + m * (12.0 * case["k"] + 8.0 * case["nev"]), "flops": 18.0 * case["atoms"] * m * (case["k"] + 1)}


# --------------------------------------------------------------------- exact
def _rmsd64(fit, ref, mass, nofit):
    """Minimum RMSD in Angstrom of every pair, [n_fit, n_ref] float64, by the largest root of the quaternion key matrix's characteristic polynomial."""
    w = torch.sqrt(mass.double() / mass.double().sum())
    centred = []
    for x in (fit, ref):
        x = x.double()
        com = (x * (mass.double() / mass.double().sum())[None, :, None]).sum(1, keepdim=True)
        centred.append((x - com) * w[None, :, None])
    a, b = centred
    e0 = a.square().sum((1, 2))[:, None] + b.square().sum((1, 2))[None, :]
    if nofit:
        d2 = torch.zeros_like(e0)
        for c in range(3):
            d2 += a[:, :, c] @ b[:, :, c].T
        return 10.0 * (e0 - 2 * d2).clamp(min=0).sqrt()
    s = [[a[:, :, c] @ b[:, :, d].T for d in range(3)] for c in range(3)]
    (sxx, sxy, sxz), (syx, syy, syz), (szx, szy, szz) = s
    c2 = torch.zeros_like(e0)
    for r in s:
        for v in r:
            c2 -= 2 * v * v
    det = sxx * (syy * szz - syz * szy) - sxy * (syx * szz - syz * szx) + sxz * (syx * szy - syy * szx)
    c1 = -8 * det
    k = [[sxx + syy + szz, syz - szy, szx - sxz, sxy - syx], [None, sxx - syy - szz, sxy + syx, szx + sxz], [None, None, -sxx + syy - szz, syz + szy], [None, None, None, -sxx - syy + szz]]
    for i in range(4):
        for j in range(i):
            k[i][j] = k[j][i]
    minor = lambda p, q, i, j: k[p][i] * k[q][j] - k[p][j] * k[q][i]  # noqa: E731
    c0 = (minor(0, 1, 0, 1) * minor(2, 3, 2, 3) - minor(0, 1, 0, 2) * minor(2, 3, 1, 3) + minor(0, 1, 0, 3) * minor(2, 3, 1, 2)
          + minor(0, 1, 1, 2) * minor(2, 3, 0, 3) - minor(0, 1, 1, 3) * minor(2, 3, 0, 2) + minor(0, 1, 2, 3) * minor(2, 3, 0, 1))
    lam = 0.5 * e0
    for _ in range(30):
        p = ((lam * lam + c2) * lam + c1) * lam + c0
        dp = (4 * lam * lam + 2 * c2) * lam + c1
        lam = lam - torch.where(dp != 0, p / dp, torch.zeros_like(p))
    return 10.0 * (e0 - 2 * lam).clamp(min=0).sqrt()


def _rms_rows(fit, ref, mass, k, nofit, full):
    out = []
    step = max(1, int(4e7) // max(1, ref.shape[0]))
    for r in range(0, fit.shape[0], step):
        d = _rmsd64(fit[r:r + step], ref, mass, nofit)
        out.append(d if full else torch.topk(d, k + 1, dim=1, largest=False).values[:, 1:])
    return torch.cat(out)


def _on_gpu(x):
    return torch.as_tensor(x, device="cuda")


def exact(case, seed):
    kind = case["kind"]
    if kind == "graph":
        return None  # a selection of the inputs: compared value by value
    if kind == "rms":
        n_fit = case["n_fit"] or case["n_ref"]
        if float(n_fit) * case["n_ref"] * (case["atoms"] + 60) > 5e11:
            return None
        s = prepare(case, seed)
        ref = _on_gpu(s["ref"])
        fit = ref if s["fit"] is None else _on_gpu(s["fit"])
        return {"d": _rms_rows(fit, ref, _on_gpu(s["mass"]), case["k"], case["nofit"], case["full"]), "i": None}
    if kind == "vec":
        n_fit = case["n_fit"] or case["n_ref"]
        if float(n_fit) * case["n_ref"] > 4.1e10:
            return None
        s = prepare(case, seed)
        ref = _on_gpu(s["ref"])
        fit = ref if s["fit"] is None else _on_gpu(s["fit"])
        if case["correlation"]:
            z = [x - x.mean(1, keepdim=True) for x in (fit, ref)]
            fit, ref = (v / v.norm(dim=1, keepdim=True) for v in z)
        out = []
        step = max(1, int(2e8) // ref.shape[0])
        rn = ref.square().sum(1)
        for r in range(0, fit.shape[0], step):
            q = fit[r:r + step]
            d2 = q.square().sum(1)[:, None] + rn[None, :] - 2 * (q @ ref.T)
            near = torch.topk(d2, case["k"] + 1, dim=1, largest=False).indices
            v = (q[:, None, :] - ref[near]).square().sum(2)
            v = v / 4 if case["correlation"] else v
            out.append(torch.sort(v, dim=1).values[:, 1:].sqrt())
        return {"d": torch.cat(out), "i": None}
    if kind == "contact":
        s = prepare(case, seed)
        x, eps = _on_gpu(s["xyz"]), case["eps"]
        half = case["atoms"] // 2
        a, b = x[:, :half], x[:, half:]
        near = []
        for r in range(0, x.shape[0], 256):
            p, q = a[r:r + 256], b[r:r + 256]
            d2 = torch.zeros(p.shape[0], p.shape[1], q.shape[1], dtype=torch.float64, device="cuda")
            for c in range(3):
                d2 += (p[:, :, None, c] - q[:, None, :, c]).square().double()
            near.append((d2.sqrt() * 10.0 < eps).reshape(p.shape[0], -1).double())
        bits = torch.cat(near)
        count = bits.sum(1)
        out = []
        for r in range(0, x.shape[0], 1024):
            d2 = count[r:r + 1024, None] + count[None, :] - 2 * (bits[r:r + 1024] @ bits.T)
            out.append(torch.topk(d2, case["k"] + 1, dim=1, largest=False).values[:, 1:].sqrt())
        return {"off": None, "idx": None, "d": torch.cat(out), "i": None}
    if kind == "eig":
        n = case["n"]
        if n > 4500:
            return None
        s = prepare(case, seed)
        col = np.repeat(np.arange(n), np.diff(s["pcol"]))
        d = np.zeros((n, n))
        d[col, s["irow"]] = d[s["irow"], col] = s["dist"]
        d = _on_gpu(d)
        k_sigma = case["k"] // 4
        if case["auto"]:
            # a landmark's first k_sigma stored distances in neighbour order
            stored = d > 0
            first = stored & (torch.cumsum(stored.to(torch.int32), 1) <= k_sigma)
            sig = (d * first).sum(1) / k_sigma
            den = 2 * sig[:, None] * sig[None, :]
        else:
            den = torch.full_like(d, 2 * s["sigma"] ** 2)
        aff = torch.where(d > 0, torch.exp(-d * d / den), torch.zeros_like(d))
        da = aff.sum(1).rsqrt()
        w, v = torch.linalg.eigh(aff * da[:, None] * da[None, :])
        w, v = w.flip(0)[:case["nev"]], v.flip(1)[:, :case["nev"]].T.contiguous()
        turn = torch.where(v @ _on_gpu(s["probe"]) < 0, -1.0, 1.0)[:, None]
        v = v * turn
        out = {"evals": w, "evecs": v, "nconv": None}
        if case["m"]:
            row = _on_gpu(s["irowB"]).long().view(case["m"], case["k"])
            db = _on_gpu(s["distB"]).view(case["m"], case["k"])
            b = torch.exp(-db * db / (2 * sig[row] ** 2 if case["auto"] else 2 * s["sigma"] ** 2))
            b = b * b.sum(1, keepdim=True).rsqrt() * da[row]
            out["ext"] = torch.stack([(b * v[x][row]).sum(1) / w[x] for x in range(case["nev"])])
        if case["auto"]:
            out["sigmas"] = sig
        return out
    # serving: the distances (the extension rests on the eigenvectors of a graph too large for a dense solver)
    sizes = _requests(case)
    x = _trajectory(case["n"] + sum(sizes), case["atoms"], _generator(seed))
    mass = torch.ones(case["atoms"], device="cuda")
    d = _rms_rows(x[case["n"]:], x[:case["n"]], mass, case["k"], False, False)
    return [{"ext": None, "d": v.contiguous(), "i": None} for v in torch.split(d, sizes)]
