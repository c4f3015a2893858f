"""The direct island solver (csrc/direct.cu) against the FP64 oracle's exact
solves, and against the conjugate-gradient path of the same entry points where
both start from the same UVs.

Tolerances: the repository's UV bar of 1e-5 of each chart's extent; where the
direct path takes an island its residual is FP64 round-off (below 1e-10). The
CG path meets its residual bar of 1e-8 in LSCM, which on a narrow strip (33 x
3 vertices) leaves 1.2e-5 of the extent, so LSCM is compared with the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import arap as O

pytestmark = pytest.mark.gpu
UV_TOL = 1e-5


def _direct(st):
    """Islands the direct path solved: a CG team counts its iterations."""
    return st["cg_iters"] == 0


def _grid(nx, ny, hole=None, seed=0, shear=0.0):
    """A jittered (nx x ny)-vertex grid patch with bumps, optionally with a
    rectangular hole, as (P, T)."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx, dtype=float), np.arange(ny, dtype=float))
    x, y = x.ravel() + shear * y.ravel(), y.ravel()
    P = np.stack([x, y, np.sin(0.7 * x) * np.cos(0.5 * y)], 1) + rng.uniform(-0.2, 0.2, (nx * ny, 3))
    idx = np.arange(nx * ny).reshape(ny, nx)
    a, b, c, d = idx[:-1, :-1], idx[:-1, 1:], idx[1:, 1:], idx[1:, :-1]
    keep = np.ones(a.shape, bool)
    if hole:
        keep[hole[1]:hole[3], hole[0]:hole[2]] = False
    T = np.concatenate([np.stack([a[keep], b[keep], c[keep]], 1), np.stack([a[keep], c[keep], d[keep]], 1)])
    used, inv = np.unique(T, return_inverse=True)
    return P[used].astype(np.float32), inv.reshape(-1, 3).astype(np.int64)


def _solve(items, direct, iters=5, semantics=None, start=None, **kw):
    from ultimate_uv_artist_b200 import _lib
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    P, T, _, vofs, tofs = concat_charts([(p, t) for p, t in items], with_uv=False)
    db = DeviceBatch(P, T, vofs, tofs, semantics=_lib.SEM_BATCH if semantics is None else semantics)
    if direct:
        db.lscm()
    else:
        _lib.check(_lib.lib().uva_lscm(C.byref(db.desc), C.byref(db.params("lscm")), db._stream()), "uva_lscm")
    torch.cuda.synchronize()
    st_l, U_l = db.island_status().copy(), db.uvs().copy()
    if start is not None:
        db.U[:db.n].copy_(torch.from_numpy(start))
    if direct:
        db.arap(iters=iters, **kw)
    else:
        prm = db.params("arap", iters=iters, **kw)
        _lib.check(_lib.lib().uva_arap(C.byref(db.desc), C.byref(prm), db._stream()), "uva_arap")
    torch.cuda.synchronize()
    return st_l, U_l, db.island_status().copy(), db.uvs().copy(), vofs


def _close(U, V, vofs):
    for a, e in zip(vofs[:-1], vofs[1:]):
        ext = max(np.ptp(V[a:e], 0).max(), 1e-12)
        assert np.abs(U[a:e] - V[a:e]).max() <= UV_TOL * ext


@pytest.mark.parametrize("shapes", [
    [(2, 2), (3, 2), (4, 4), (5, 3), (16, 1 + 1), (17, 2)],              # one block, its edge, two blocks
    [(4, 8), (3, 11), (31, 2), (32, 2), (33, 3)],                        # remainders of 16 rows
    [(200, 3), (3, 200), (40, 41), (64, 64)],                            # long, wide, square
    [(90, 91), (128, 128)],                                              # above 8,192 vertices; exactly 16,384
], ids=["blocks", "remainders", "aspect", "large"])
def test_direct_matches_exact_solves(cuda, shapes):
    items = [_grid(w, h, seed=k) for k, (w, h) in enumerate(shapes)]
    ref = [(p.astype(np.float64), t, O.lscm(p.astype(np.float64), t)) for p, t in items]
    start = np.concatenate([u for _, _, u in ref])
    st_l, U_l, st_a, U_a, vofs = _solve(items, True, start=start)
    assert _direct(st_l).all() and _direct(st_a).all()
    assert (st_l["flags"] == 0).all() and (st_a["flags"] == 0).all()
    assert (st_l["resid"] <= 1e-10).all() and (st_a["resid"] <= 1e-10).all()
    _close(U_l, start, vofs)
    r = O.BatchRef(ref)
    r.arap(5, line_search=True)
    _close(U_a, r.U, vofs)


def test_direct_matches_the_oracle(cuda):
    items = [_grid(37, 29, seed=1), _grid(30, 30, hole=(10, 10, 20, 20), seed=2), _grid(70, 5, seed=3, shear=0.5)]
    _, U_l, _, U_a, vofs = _solve(items, True, iters=6)
    ref = [(p.astype(np.float64), t, O.lscm(p.astype(np.float64), t)) for p, t in items]
    assert O.uv_rel_error(U_l, np.concatenate([u for _, _, u in ref]), vofs) < UV_TOL
    r = O.BatchRef(ref)
    r.arap(6, line_search=True)
    assert O.uv_rel_error(U_a, r.U, vofs) < UV_TOL


def test_singular_and_wide_islands_keep_cg(cuda):
    """Two components, an island whose skyline is wider than 15 blocks and one
    above 16,384 vertices take the CG path, the ones around them the direct
    path; ARAP and LSCM results match an all-CG run."""
    from ultimate_uv_artist_b200 import _lib
    g1, g2 = _grid(9, 9, seed=4), _grid(8, 12, seed=5)
    two = (np.concatenate([g1[0], g2[0] + 30]), np.concatenate([g1[1], g2[1] + len(g1[0])]))
    # a hub joined to 300 outer vertices: one breadth-first level of 300
    ang = np.linspace(0, 2 * np.pi, 301)[:-1]
    hub = (np.concatenate([[[0, 0, 0.1]], np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1)]).astype(np.float32),
           np.stack([np.zeros(300, int), 1 + np.arange(300), 1 + (np.arange(300) + 1) % 300], 1))
    items = [_grid(12, 12, seed=6), two, hub, _grid(129, 128, seed=7), _grid(20, 20, seed=8)]
    start = np.concatenate([p[:, :2].astype(np.float64) for p, _ in items])
    a, b = _solve(items, True, iters=4, start=start), _solve(items, False, iters=4, start=start)
    took = _direct(a[2])
    assert took[0] and took[4] and not took[1] and not took[2] and not took[3]
    for k in (0, 2, 3, 4):      # the unpinned component of the second island is not determined
        s = slice(a[4][k], a[4][k + 1])
        assert np.abs(a[3][s] - b[3][s]).max() <= UV_TOL * np.ptp(b[3][s], 0).max()
    assert (a[2]["resid"] <= 2e-7 * 1.001).all() and ((a[2]["flags"] & _lib.ST_BADCLASS) == 0).all()


@pytest.mark.parametrize("kw", [dict(line_search=False), dict(energy_tol=1e-3), dict(fold_step=True), dict(iters=2)],
                         ids=["free", "energy", "fold", "few"])
def test_options_match_cg(cuda, kw):
    from ultimate_uv_artist_b200 import _lib
    kw = dict(kw)
    iters = kw.pop("iters", 12)
    sem = _lib.SEM_PARAM if "energy_tol" in kw else _lib.SEM_BATCH
    items = [_grid(14, 15, seed=9), _grid(33, 8, seed=10)]
    start = np.concatenate([O.lscm(p.astype(np.float64), t) for p, t in items])
    a, b = (_solve(items, d, iters, sem, start, **kw) for d in (True, False))
    assert (_direct(a[2]) == (iters >= 3)).all()     # short calls keep CG: no factor to pay for
    assert np.array_equal(a[2]["outer_iters"], b[2]["outer_iters"])
    assert np.array_equal(a[2]["flags"], b[2]["flags"])
    _close(a[3], b[3], a[4])


def test_small_scratch_keeps_cg(cuda):
    """Parts too small for their islands' factors leave the islands to CG."""
    from ultimate_uv_artist_b200 import _lib
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    P, T, _, vofs, tofs = concat_charts([_grid(40, 40, seed=11), _grid(6, 6, seed=12)], with_uv=False)
    db = DeviceBatch(P, T, vofs, tofs)
    half = db._direct_parts // 4 // 256 * 256
    db._direct_parts = half
    db.direct_ofs.copy_(torch.from_numpy(half))
    db.lscm()
    db.arap(iters=4)
    st = db.island_status()
    assert not _direct(st).any() and (st["resid"] <= 2e-7 * 1.001).all() and (st["flags"] & 3 == 0).all()
