"""Which launches the factors get and which CG (k_choose in csrc/direct.cu):
the batches on which either was measured faster take that one, and both give
the same UVs: LSCM within 1e-5 and ARAP from the same start within 1e-5 of a
chart's extent, the repository's UV bar (residuals of 1e-8 and 2e-7)."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_direct import UV_TOL, _grid

pytestmark = pytest.mark.gpu


def _irregular(seed, n):
    """A bumped disk of n random points, Delaunay triangles."""
    from scipy.spatial import Delaunay
    rng = np.random.default_rng(seed)
    r, a = np.sqrt(rng.random(n)), rng.uniform(0, 2 * np.pi, n)
    p = np.stack([r * np.cos(a), r * np.sin(a)], 1)
    t = Delaunay(p).simplices
    e1, e2 = p[t[:, 1]] - p[t[:, 0]], p[t[:, 2]] - p[t[:, 0]]
    area = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
    t = np.where((area > 0)[:, None], t, t[:, [0, 2, 1]])[np.abs(area) > 1e-7]
    used, inv = np.unique(t, return_inverse=True)
    p = p[used]
    return (np.concatenate([p, 0.3 * np.sin(3 * p[:, :1])], 1).astype(np.float32), inv.reshape(-1, 3).astype(np.int64))


def _batch(items):
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    P, T, _, vofs, tofs = concat_charts(items, with_uv=False)
    return DeviceBatch(P, T, vofs, tofs), vofs


def _by_cg(db, kind, **kw):
    from ultimate_uv_artist_b200 import _lib
    prm = db.params(kind, **kw)
    _lib.check(getattr(_lib.lib(), "uva_" + kind)(C.byref(db.desc), C.byref(prm), db._stream()), kind)


def _same(U, V, vofs):
    for a, e in zip(vofs[:-1], vofs[1:]):
        assert np.abs(U[a:e] - V[a:e]).max() <= UV_TOL * max(np.ptp(V[a:e], 0).max(), 1e-12)


# (charts, iterations, LSCM by factors, ARAP by factors)
CASES = {
    "one_small": ([(20, 20)], 20, True, True),
    "one_large_few_iterations": ([(88, 90)], 3, True, True),
    "one_large": ([(88, 90)], 20, True, True),                        # too near to call: factors
    "some_large": ([(88, 90)] * 60 + [(40, 40)] * 100, 20, True, False),   # the factors' chains, out of L2
    "above_the_cta_class": ([(100, 100)], 20, True, True),            # CG's vectors would be in global memory
    "many_mid": ([(30, 30)] * 700, 8, True, True),
    "large_among_many": ([(88, 90)] * 8 + [(30, 30)] * 3000, 20, True, True),   # the others fill the launch
    "tiny": ([(4, 5)] * 20000, 10, False, True),
    "few_tiny": ([(4, 5)] * 50, 4, True, True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_choice_and_results(cuda, name):
    shapes, iters, lscm_f, arap_f = CASES[name]
    made = {s: _grid(*s, seed=3) for s in set(shapes)}
    db, vofs = _batch([made[s] for s in shapes])
    db.lscm()
    assert ((db.island_status()["cg_iters"] == 0) == lscm_f).all()
    U_l = db.uvs().copy()
    _by_cg(db, "lscm")
    _same(U_l, db.uvs(), vofs)
    start = torch.from_numpy(U_l)
    db.U[:db.n].copy_(start)
    db.arap(iters=iters)
    st = db.island_status()
    assert ((st["cg_iters"] == 0) == arap_f).all()
    assert (st["flags"] == 0).all() and (st["outer_iters"] == iters).all()
    assert (st["resid"] <= 1e-7 * 1.001).all()      # in place of a factor CG takes half the tolerance
    U_a = db.uvs().copy()
    db.U[:db.n].copy_(start)
    g = db.step_graph(setup=False, lscm=False, arap_iters=iters)     # the same choice in a captured call
    g.launch()
    torch.cuda.synchronize()
    assert np.array_equal(db.uvs(), U_a)
    g.close()


@pytest.mark.parametrize("kind", ["lscm", "arap"])
def test_irregular_charts_without_a_factor(cuda, kind):
    """Charts of one size, some of them without a factor: a launch of factors
    before CG would only add to it, so all take CG."""
    from ultimate_uv_artist_b200.device import direct_parts
    db, vofs = _batch([_irregular(s, 1300) for s in range(40)])
    info = db.band[db.n + db.n // 16 + db.nc:][:4 * db.nc].view(-1, 4).cpu().numpy()
    order = db.plan.order
    room = np.diff(direct_parts(np.diff(vofs), db.direct_slots), axis=1)[0][:db.nc]
    need = (info[order, 1] + 256) * 2048 + (np.diff(vofs)[order] + 15) // 16 * 768
    takes = (info[order, 0] & 1 == 1) & (need <= room)
    assert 0 < takes.sum() < 40
    if kind == "arap":
        db.lscm()
        db.arap(iters=8)
    else:
        db.lscm()
    st = db.island_status()
    assert (st["cg_iters"] > 0).all() and (st["flags"] == 0).all()


def test_tight_tolerance_keeps_factors(cuda):
    """At 1e-10 CG takes half as many iterations again."""
    db, _ = _batch([_grid(88, 90, seed=3)])
    db.lscm()
    db.arap(iters=20, tol=1e-10)
    assert (db.island_status()["cg_iters"] == 0).all()
