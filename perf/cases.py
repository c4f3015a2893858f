"""Performance cases of the framework: what a program that unwraps meshes has
it do, through the public entry points, from one chart to a whole atlas.

Kinds (``case["kind"]``):

* ``unwrap``    charts on the host -> ``gpu.Batch`` -> ``lscm`` -> ``arap``:
                the call an unwrapper makes for a new set of charts, uploads,
                topology plan and set-up included;
* ``lscm``      ``Batch.lscm`` of a batch that is on the device already;
* ``arap``      ``Batch.arap`` from the batch's LSCM layout (charts refined
                again after an edit, or refined further);
* ``validate``  ``validate.validate_uvs`` of an exported atlas on the host;
* ``energy``    value and gradients of the differentiable distortion energy;
* ``report``    ``metrics.distortion_report`` of an atlas on the host;
* ``pack``      ``pack.pack`` of the solved charts.

Charts are disks cut from square grids (a random diagonal in every cell, so
vertex degrees run from 3 to 8), jittered in the plane and displaced by
Gaussian bumps. A chart's size is the triangle count of its square grid, of
which the disk keeps about pi / 4; sizes are spread over the logarithm of the
stated range, as the islands of a scan are. The sizes follow from the case, all
else from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ultimate_uv_artist_b200 import synth
from ultimate_uv_artist_b200.energy import distortion_energy
from ultimate_uv_artist_b200.engine import gpu, metrics, pack, validate


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a single chart of the size of one 50 x 50 patch: the latency of one call
        {"name": "unwrap_one_chart", "kind": "unwrap", "islands": 1, "tmin": 6100, "tmax": 6100, "iters": 10},
        # a low-poly prop: a few dozen small charts, about 12,000 triangles
        {"name": "unwrap_low_poly", "kind": "unwrap", "islands": 61, "tmin": 20, "tmax": 1000, "iters": 8},
        # a dense scan, thousands of uneven charts: the headline workload, host to result
        {"name": "unwrap_scan", "kind": "unwrap", "islands": 2000, "tmin": 20, "tmax": 20000, "iters": 20},
        # the two solves of the same workload on a resident batch
        {"name": "lscm_scan", "kind": "lscm", "islands": 2000, "tmin": 20, "tmax": 20000},
        {"name": "arap_scan", "kind": "arap", "islands": 2000, "tmin": 20, "tmax": 20000, "iters": 20},
        # a character: one very large chart among small ones (whole-GPU team)
        {"name": "arap_large_chart", "kind": "arap", "islands": 60, "tmin": 20, "tmax": 3000, "big": 153000, "iters": 8},
        # the exported atlas of a game prop, checked against its input mesh
        {"name": "validate_prop", "kind": "validate", "islands": 301, "tris": 72, "atlas": 2048, "padding": 4,
         "preserve": True},
        # a million exported triangles at 4096 texels
        {"name": "validate_atlas", "kind": "validate", "islands": 5000, "tris": 200, "atlas": 4096, "padding": 4,
         "preserve": False},
        # optimisation loops on the ARAP energy: UV gradients of a few charts
        {"name": "energy_arap_few", "kind": "energy", "islands": 24, "tmin": 600, "tmax": 12000, "energy": 0,
         "grad_positions": False},
        # symmetric Dirichlet energy of millions of triangles, UV and position gradients
        {"name": "energy_dirichlet_scan", "kind": "energy", "islands": 512, "tmin": 640, "tmax": 64000, "energy": 1,
         "grad_positions": True},
        # the distortion statistics of a finished atlas
        {"name": "report_atlas", "kind": "report", "islands": 600, "tmin": 20, "tmax": 20000},
        # a few hundred charts into one page, the packer's default schedule
        {"name": "pack_charts", "kind": "pack", "islands": 180, "tmin": 20, "tmax": 4000, "atlas": 2048, "padding": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["unwrap", "lscm", "lscm", "arap", "arap", "validate", "energy", "energy", "report", "pack"])
    if kind in ("unwrap", "lscm", "arap"):
        n = _log(rng, 1, 1200)
        case = {"kind": kind, "islands": n, "tmin": _log(rng, 20, 200) if n >= 16 else _log(rng, 300, 600),
                "tmax": _log(rng, 700, 24000)}
        if kind != "lscm":
            case["iters"] = rng.randint(4, 20)
        if kind == "arap" and rng.random() < 0.25:
            case.update(islands=_log(rng, 1, 100), big=_log(rng, 45000, 140000))
        return case
    if kind == "validate":
        return {"kind": kind, "islands": _log(rng, 200, 4000), "tris": rng.choice([18, 50, 98, 128, 200]),
                "atlas": rng.choice([1024, 2048, 4096]), "padding": rng.choice([2, 4]),
                "preserve": rng.random() < 0.5}
    if kind == "energy":
        return {"kind": kind, "islands": _log(rng, 1, 400), "tmin": _log(rng, 300, 1000),
                "tmax": _log(rng, 2000, 60000), "energy": rng.randint(0, 1), "grad_positions": rng.random() < 0.5}
    if kind == "report":
        return {"kind": kind, "islands": _log(rng, 1, 500), "tmin": _log(rng, 20, 200),
                "tmax": _log(rng, 400, 20000)}
    return {"kind": kind, "islands": _log(rng, 20, 150), "tmin": 20, "tmax": _log(rng, 200, 3000),
            "atlas": rng.choice([1024, 2048]), "padding": rng.choice([2, 4])}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _disk(cells):
    """A disk of whole grid cells with a random diagonal in each: the grid
    rows and columns of its vertices and its triangles."""
    rng = np.random.default_rng(7919 + cells)
    nx = cells + 1
    cc = (np.arange(cells) + 0.5) / cells * 2 - 1
    keep = (cc[None, :] ** 2 + cc[:, None] ** 2) <= 1.0
    idx = np.arange(nx * nx, dtype=np.int64).reshape(nx, nx)
    a, b, c, d = idx[:-1, :-1][keep], idx[:-1, 1:][keep], idx[1:, 1:][keep], idx[1:, :-1][keep]
    par = (rng.random(len(a)) < 0.5)[:, None]
    t1 = np.where(par, np.stack([a, b, c], -1), np.stack([a, b, d], -1))
    t2 = np.where(par, np.stack([a, c, d], -1), np.stack([b, c, d], -1))
    F = np.stack([t1, t2], 1).reshape(-1, 3)
    used, inv = np.unique(F, return_inverse=True)
    return used // nx, used % nx, np.ascontiguousarray(inv.reshape(-1, 3).astype(np.int64))


def _chart(rng, tris):
    """(P float32 (n, 3), T int64 (t, 3)) of a square grid of ``tris`` triangles."""
    cells = max(2, int(round(math.sqrt(tris / 2))))
    row, col, T = _disk(cells)
    s = np.linspace(-1.0, 1.0, cells + 1)
    c = rng.uniform(-1.0, 1.0, (2, 8))
    amp, sg = rng.uniform(0.0, 0.5, 8), rng.uniform(0.15, 0.45, 8)
    g = np.exp(-((s[None, :, None] - c[:, None, :]) ** 2) / (2 * sg * sg))
    z = (g[0] * amp) @ g[1].T
    j = rng.uniform(-0.3 / cells, 0.3 / cells, (2, len(row)))
    P = np.stack([s[col] + j[0], s[row] + j[1], z[row, col]], 1)
    return P.astype(np.float32), T


def _charts(case, seed):
    fixed = np.random.default_rng([case["islands"], case["tmin"], case["tmax"]])   # a case's sizes; the seed orders them
    sizes = np.exp(fixed.uniform(math.log(case["tmin"]), math.log(case["tmax"]), case["islands"]))
    if case.get("big"):
        sizes[0] = case["big"]
    rng = np.random.default_rng(seed)
    return [_chart(rng, t) for t in rng.permutation(sizes)]


def _whole(charts):
    """Positions, triangles (global ids) and the chart of each triangle."""
    nv = np.cumsum([0] + [len(P) for P, _ in charts])
    F = np.concatenate([T + o for (_, T), o in zip(charts, nv)])
    lab = np.repeat(np.arange(len(charts)), [len(T) for _, T in charts])
    return np.concatenate([P for P, _ in charts]), F, lab, nv


def _atlas(case, seed):
    return synth.validation_atlas(seed=seed, islands=case["islands"], tris_per_island=case["tris"],
                                  atlas=case["atlas"], padding=case["padding"])[:3]


def _energy_inputs(case, seed):
    """Charts, positions and flip-free UVs some way from the energy's minimum
    (an affine image of the projection)."""
    charts = _charts(case, seed)
    P, F, lab, nv = _whole(charts)
    rng = np.random.default_rng([seed, 1])
    m = np.eye(2) + rng.uniform(-0.2, 0.2, (len(charts), 2, 2))
    of = np.repeat(np.arange(len(charts)), np.diff(nv))
    U = np.einsum("nij,nj->ni", m[of], P[:, :2].astype(np.float64))
    return charts, P, F, lab, U


def _report_inputs(case, seed):
    charts = _charts(case, seed)
    P, F, lab, nv = _whole(charts)
    rng = np.random.default_rng([seed, 2])
    of = np.repeat(np.arange(len(charts)), np.diff(nv))
    size = rng.uniform(0.8, 1.25, len(charts)) * 0.5 / math.sqrt(len(charts))
    mirror = np.where(rng.random(len(charts)) < 0.02, -1.0, 1.0)
    UV = P[:, :2] * size[of][:, None] + rng.uniform(0.1, 0.9, (len(charts), 2))[of]
    UV[:, 0] *= mirror[of]
    return P, F, UV.astype(np.float32), lab.astype(np.int32)


def prepare(case, seed):
    """What the calling program holds before the call."""
    kind = case["kind"]
    if kind == "unwrap":
        return {"case": case, "charts": [(P, T, None) for P, T in _charts(case, seed)]}
    if kind in ("lscm", "arap"):
        b = gpu.Batch([(P, T, None) for P, T in _charts(case, seed)])
        U0 = b.lscm().clone() if kind == "arap" else None
        return {"case": case, "batch": b, "U0": U0}
    if kind == "validate":
        V, F, UV = _atlas(case, seed)
        return {"case": case, "V": V, "F": F, "UV": UV}
    if kind == "energy":
        charts, _, _, _, U = _energy_inputs(case, seed)
        b = gpu.Batch([(P, T, None) for P, T in charts])
        Ut = torch.from_numpy(U).to(b.dev).requires_grad_(True)
        Pt = b.db.P[:b.n].clone().requires_grad_(bool(case["grad_positions"]))
        return {"case": case, "batch": b, "U": Ut, "P": Pt}
    if kind == "report":
        V, F, UV, lab = _report_inputs(case, seed)
        return {"case": case, "V": V, "F": F, "UV": UV, "islands": lab}
    rng = np.random.default_rng([seed, 3])
    charts = []
    for P, T in _charts(case, seed):
        turn, k = rng.uniform(0, 2 * math.pi), rng.uniform(0.5, 1.0, 2) * math.sqrt(len(T))
        c, s = math.cos(turn), math.sin(turn)
        charts.append(((P[:, :2].astype(np.float64) * k) @ np.array([[c, s], [-s, c]]), T))
    return {"case": case, "charts": charts}


# ------------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "unwrap":
        b = gpu.Batch(state["charts"])
        b.lscm()
        return b.arap(iters=case["iters"])
    if kind == "lscm":
        return state["batch"].lscm()
    if kind == "arap":
        b = state["batch"]
        b.U = state["U0"]
        return b.arap(iters=case["iters"])
    if kind == "validate":
        V, F, UV = state["V"], state["F"], state["UV"]
        src = {"in_v": V, "in_f": F} if case["preserve"] else {}
        report, problems = validate.validate_uvs(V, F, UV, atlas=case["atlas"], padding=case["padding"], **src)
        return {"report": report, "problems": problems}
    if kind == "energy":
        U, P = state["U"], state["P"]
        e = distortion_energy(state["batch"].db, U, P, case["energy"])
        wrt = (U, P) if case["grad_positions"] else (U,)
        return [e.detach(), *torch.autograd.grad(e.sum(), wrt)]
    if kind == "report":
        return metrics.distortion_report(state["V"], state["F"], state["UV"], state["islands"])
    uvs, info = pack.pack(state["charts"], atlas=case["atlas"], padding=case["padding"])
    return {"uv": np.concatenate(uvs), "scale": info["texel_scale_grid"], "occupancy": info["plan_occupancy"]}


# ------------------------------------------------------------------ the work of a pass
def _mean_tris(case):
    lo, hi = case["tmin"], case["tmax"]
    one = (hi - lo) / math.log(hi / lo) if hi > lo else lo
    return math.pi / 4 * (one * case["islands"] + (case.get("big") or 0))


def work(case):
    """Compulsory traffic and arithmetic: inputs read once, outputs written
    once; per triangle about 60 operations for a conformal system, 200 for an
    ARAP iteration (rotation, right-hand side, one product with the matrix),
    250 for an energy with its gradient, 400 for the statistics."""
    kind = case["kind"]
    if kind == "validate":
        t = case["islands"] * case["tris"]
        n = 0.65 * t
        return {"bytes": 20 * n + 24 * t + t + case["atlas"] ** 2 / 8, "flops": 100 * t}
    t = _mean_tris(case)
    n = 0.53 * t
    if kind == "unwrap":
        return {"bytes": 24 * t + 12 * n + 8 * n, "flops": (60 + 200 * case["iters"]) * t}
    if kind == "lscm":
        return {"bytes": 12 * t + 12 * n + 8 * n, "flops": 60 * t}
    if kind == "arap":
        return {"bytes": 12 * t + 12 * n + 16 * n, "flops": 200 * case["iters"] * t}
    if kind == "energy":
        p = 24 if case["grad_positions"] else 0
        return {"bytes": 12 * t + (16 + 24 + 16 + p) * n, "flops": 250 * t}
    if kind == "report":
        return {"bytes": 24 * t + 4 * t + 20 * n, "flops": 400 * t}
    return {"bytes": 24 * t + 32 * n, "flops": 100 * t}


# ------------------------------------------------------------------ 64-bit values
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _frames(P, T):
    """(x1, x2, y2) of each triangle in its own plane, corner 0 at the origin."""
    e1, e2 = P[T[:, 1]] - P[T[:, 0]], P[T[:, 2]] - P[T[:, 0]]
    x1 = e1.norm(dim=1)
    n = torch.linalg.cross(e1, e2).norm(dim=1)
    return x1, (e1 * e2).sum(1) / x1, n / x1


def _half_cots(x1, x2, y2):
    c = torch.stack([torch.stack([0 * x1, 0 * x1], 1), torch.stack([x1, 0 * x1], 1), torch.stack([x2, y2], 1)], 1)
    w = []
    for k in range(3):
        a, b = c[:, (k + 1) % 3] - c[:, k], c[:, (k + 2) % 3] - c[:, k]
        cr = (a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]).abs()
        w.append(0.5 * ((a * b).sum(1) / cr).clamp(-1e4, 1e4))
    return c, torch.stack(w, 1)


def _far_pair(P, T):
    """The two pinned boundary vertices: farthest from the boundary's centre,
    then farthest from that one."""
    a, b = T.reshape(-1), T[:, [1, 2, 0]].reshape(-1)
    n = int(T.max()) + 1
    key, rev = a * n + b, b * n + a
    bv = torch.unique(a[~torch.isin(key, rev)])
    Q = P[bv]
    i = int(((Q - Q.mean(0)) ** 2).sum(1).argmax())
    j = int(((Q - Q[i]) ** 2).sum(1).argmax())
    return int(bv[i]), int(bv[j])


def _exact_lscm(P, T):
    """Least-squares conformal map: per triangle |sum_k W_k u_k|^2 / (4 area)
    over complex vertex positions u, two vertices fixed."""
    n = len(P)
    x1, x2, y2 = _frames(P, T)
    z = torch.stack([torch.zeros_like(x1) + 0j, x1 + 0j, torch.complex(x2, y2)], 1)
    W = (z[:, [2, 0, 1]] - z[:, [1, 2, 0]]) / (2 * x1 * y2).sqrt()[:, None]
    H = torch.zeros((n, n), dtype=torch.complex128, device=P.device)
    for k in range(3):
        for m in range(3):
            H.view(-1).index_add_(0, T[:, k] * n + T[:, m], W[:, k].conj() * W[:, m])
    p0, p1 = _far_pair(P, T)
    u1 = float((P[p1] - P[p0]).norm())
    rhs = -H[:, p1].clone() * u1
    for p, u in ((p0, 0.0), (p1, u1)):      # the fixed rows and columns become the identity
        H[p, :] = 0
        H[:, p] = 0
        H[p, p] = 1
        rhs[p] = u
    x = torch.cholesky_solve(rhs[:, None], torch.linalg.cholesky(H))[:, 0]
    return torch.stack([x.real, x.imag], 1)


def _exact_arap(charts, U, iters):
    """ARAP local / global iterations with the flip-safe step; vertex 0 of a
    chart softly pinned with the batch's largest |weight|. Charts in groups:
    the local steps of a group together, an explicit inverse per chart."""
    dev = _dev()
    geo = []
    for P, T in charts:
        P, T = torch.from_numpy(P).to(dev, torch.float64), torch.from_numpy(T).to(dev)
        c, w = _half_cots(*_frames(P, T))
        geo.append((len(P), T, c, w))
    wpin = max(float(g[3].abs().max()) for g in geo)
    out, at = [], 0
    while at < len(geo):
        end, cells = at, 0
        while end < len(geo) and (end == at or cells + geo[end][0] ** 2 <= 4e8):
            cells += geo[end][0] ** 2
            end += 1
        group = geo[at:end]
        ofs = np.cumsum([0] + [g[0] for g in group]).tolist()
        base = sum(len(u) for u in out)
        X = U[base:base + ofs[-1]].clone()
        T = torch.cat([g[1] + o for g, o in zip(group, ofs)])
        c, w = torch.cat([g[2] for g in group]), torch.cat([g[3] for g in group])
        tri = torch.repeat_interleave(torch.arange(len(group), device=dev),
                                      torch.tensor([len(g[1]) for g in group], device=dev))
        of = torch.repeat_interleave(torch.arange(len(group), device=dev), torch.tensor(np.diff(ofs), device=dev))
        inv = []
        for n, Ti, _, wi in group:
            L = torch.zeros((n, n), dtype=torch.float64, device=dev)
            for k in range(3):
                i, j = Ti[:, (k + 1) % 3], Ti[:, (k + 2) % 3]
                for r, s, sign in ((i, j, -1), (j, i, -1), (i, i, 1), (j, j, 1)):
                    L.view(-1).index_add_(0, r * n + s, sign * wi[:, k])
            L[0, 0] += wpin
            inv.append(torch.cholesky_inverse(torch.linalg.cholesky(L)))
        first = torch.tensor(ofs[:-1], device=dev)
        for _ in range(iters):
            d1, d2 = X[T[:, 1]] - X[T[:, 0]], X[T[:, 2]] - X[T[:, 0]]
            a = d1 / c[:, 1, :1]
            b = (d2 - a * c[:, 2, :1]) / c[:, 2, 1:]
            ca, cb = a[:, 0] + b[:, 1], a[:, 1] - b[:, 0]
            h = torch.hypot(ca, cb)
            co, si = torch.where(h > 0, ca / h, 1.0), torch.where(h > 0, cb / h, 0.0)
            rhs = torch.zeros_like(X)
            for k in range(3):
                i, j = (k + 1) % 3, (k + 2) % 3
                e = c[:, i] - c[:, j]
                v = w[:, k:k + 1] * torch.stack([co * e[:, 0] - si * e[:, 1], si * e[:, 0] + co * e[:, 1]], 1)
                rhs.index_add_(0, T[:, i], v)
                rhs.index_add_(0, T[:, j], -v)
            rhs[first] += wpin * X[first]
            Y = torch.cat([m @ rhs[p:q] for m, p, q in zip(inv, ofs[:-1], ofs[1:])])
            D = Y - X
            g1, g2 = D[T[:, 1]] - D[T[:, 0]], D[T[:, 2]] - D[T[:, 0]]
            C = d1[:, 0] * d2[:, 1] - d2[:, 0] * d1[:, 1]
            B = d1[:, 0] * g2[:, 1] + g1[:, 0] * d2[:, 1] - d2[:, 0] * g1[:, 1] - g2[:, 0] * d1[:, 1]
            A = g1[:, 0] * g2[:, 1] - g2[:, 0] * g1[:, 1]
            flat = A.abs() < 1e-30
            sq = (B * B - 4 * A * C).sqrt()
            roots = torch.stack([(-B - sq) / (2 * A), (-B + sq) / (2 * A)], 1)
            roots = torch.where(flat[:, None], torch.where(B < 0, -C / B, -1.0)[:, None], roots)
            roots = torch.where((roots > 0) & (C > 0)[:, None], roots, 1e30)
            t = torch.full((len(group),), 1e30, dtype=torch.float64, device=dev)
            t.scatter_reduce_(0, tri, roots.min(1).values, "amin")
            X = X + D * (0.9 * t).clamp(max=1.0)[of][:, None]
        out.append(X)
        at = end
    return torch.cat(out)


def _exact_solve(case, seed):
    charts = _charts(case, seed)
    if max(len(P) for P, _ in charts) > 12000 or sum(len(P) ** 3 for P, _ in charts) > 8e13:
        return None
    dev = _dev()
    U = torch.cat([_exact_lscm(torch.from_numpy(P).to(dev, torch.float64), torch.from_numpy(T).to(dev))
                   for P, T in charts])
    return U if case["kind"] == "lscm" else _exact_arap(charts, U, case["iters"])


def _exact_energy(case, seed):
    charts, P, F, lab, U = _energy_inputs(case, seed)
    dev = _dev()
    P = torch.from_numpy(P).to(dev, torch.float64).requires_grad_(True)
    U = torch.from_numpy(U).to(dev).requires_grad_(True)
    F, lab = torch.from_numpy(F).to(dev), torch.from_numpy(lab).to(dev)
    x1, x2, y2 = _frames(P, F)
    a = (U[F[:, 1]] - U[F[:, 0]]) / x1[:, None]
    b = (U[F[:, 2]] - U[F[:, 0]] - a * x2[:, None]) / y2[:, None]
    fro, area = (a * a).sum(1) + (b * b).sum(1), 0.5 * x1 * y2
    det = a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]
    if case["energy"] == 0:     # |J - R|^2 = |J|^2 - 2 (s1 + s2) + 2, s1 + s2 = |(j00 + j11, j10 - j01)|
        f = fro - 2 * torch.hypot(a[:, 0] + b[:, 1], a[:, 1] - b[:, 0]) + 2
    else:
        f = fro + fro / (det * det) - 4
    e = torch.zeros(len(charts), dtype=torch.float64, device=dev).index_add_(0, lab, area * f)
    wrt = (U, P) if case["grad_positions"] else (U,)
    return [e.detach(), *torch.autograd.grad(e.sum(), wrt)]


def _wquantile(x, w, q):
    i = torch.argsort(x)
    c = torch.cumsum(w[i], 0)
    k = int(torch.searchsorted(c, q * c[-1]))
    return float(x[i][min(k, len(x) - 1)])


def _corner_angles(p):
    out = []
    for k in range(3):
        u, v = p[:, (k + 1) % 3] - p[:, k], p[:, (k + 2) % 3] - p[:, k]
        out.append(torch.arccos(((u * v).sum(1) / (u.norm(dim=1) * v.norm(dim=1))).clamp(-1, 1)))
    return torch.stack(out, 1)


def _exact_report(case, seed):
    V, F, UV, lab = _report_inputs(case, seed)
    dev = _dev()
    P, U = torch.from_numpy(V).to(dev, torch.float64), torch.from_numpy(UV).to(dev, torch.float64)
    F, lab = torch.from_numpy(F).to(dev), torch.from_numpy(lab).to(dev).long()
    x1, x2, y2 = _frames(P, F)
    d1, d2 = U[F[:, 1]] - U[F[:, 0]], U[F[:, 2]] - U[F[:, 0]]
    a = d1 / x1[:, None]
    b = (d2 - a * x2[:, None]) / y2[:, None]
    q = 0.5 * torch.hypot(a[:, 0] + b[:, 1], a[:, 1] - b[:, 0])
    r = 0.5 * torch.hypot(a[:, 0] - b[:, 1], a[:, 1] + b[:, 0])
    s1, s2, a3 = q + r, (q - r).abs(), 0.5 * x1 * y2
    sa = 0.5 * (d1[:, 0] * d2[:, 1] - d1[:, 1] * d2[:, 0])
    w = a3 / a3.sum()
    scale2 = sa.abs().sum() / a3.sum()
    ok = sa.abs() >= 1e-2 / 8192.0 ** 2
    live = w * ok
    lg = torch.log2((s1 * s2 / scale2).clamp(min=1e-30)).abs()
    n = int(lab.max()) + 1
    add = lambda v: torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, lab, v)  # noqa: E731
    i3, iu, up, dn = add(a3), add(sa.abs()), add(a3 * (sa > 0)), add(a3 * (sa < 0))
    lc = torch.log2((s1 * s2 / (iu / i3)[lab]).clamp(min=1e-30)).abs()
    dom = torch.where(up >= dn, 1.0, -1.0)
    flip = ok & (sa.sign() != dom[lab])
    ang = (_corner_angles(P[F]) - _corner_angles(U[F])).abs().mean(1) * (180 / math.pi)
    an = s1 / s2
    st2 = (s1 * s1 + s2 * s2) / 2 / scale2
    dens = torch.log2((iu / i3 / scale2).sqrt()).abs()
    sel = lambda v: (v[ok], live[ok])  # noqa: E731
    return {"triangles": None, "collapsed_uv_triangles": None, "flipped_triangles": None, "mirrored_islands": None,
            "collapsed_uv_area_fraction": float((w * ~ok).sum()),
            "anisotropy_mean": float((an * live).sum() / live.sum()), "anisotropy_p95": _wquantile(*sel(an), 0.95),
            "angle_error_deg_mean": float((ang * w).sum() / w.sum()),
            "density_log2_dev_mean": float((lg * live).sum() / live.sum()),
            "density_ratio_p95": 2 ** _wquantile(*sel(lg), 0.95),
            "stretch_L2": float(((st2 * live).sum() / live.sum()).sqrt()),
            "chart_area_log2_dev_mean": float((lc * live).sum() / live.sum()),
            "chart_area_ratio_p95": 2 ** _wquantile(*sel(lc), 0.95),
            "flipped_area_fraction": float((w * flip).sum()),
            "island_density_ratio_p95": 2 ** _wquantile(dens, i3, 0.95)}


def exact(case, seed):
    """The floating outputs of ``run`` in 64 bits, by plain dense torch; None
    where that takes too long (a chart above 12,000 vertices) and for the
    validation's and the packer's outputs, which are counts and placements."""
    kind = case["kind"]
    if kind in ("unwrap", "lscm", "arap"):
        return _exact_solve(case, seed)
    if kind == "energy":
        return _exact_energy(case, seed)
    return _exact_report(case, seed) if kind == "report" else None
