"""The coarse operators that the set-up leaves out of islands with a factor,
built by the first solve that gives such an island to CG: the same UVs, bit
for bit, as a batch without an elimination order, whose set-up builds them
all. Islands of each size class (aggregates of 64 rows and more, operators in
shared and in global memory, one above 16,384 vertices), ARAP calls of few
iterations (twice: built once), LSCM without the factor's scratch, a captured
call, and a factor solve before."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = {
    "small": [(2, 2), (5, 7), (16, 16), (16, 17), (30, 40)],
    "cta": [(45, 46), (64, 65), (90, 92), (10, 10)],
    "global": [(110, 112), (128, 128), (20, 20)],
    "wide": [(129, 128), (30, 30)],
}


def _grid(nx, ny, seed):
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx, dtype=float), np.arange(ny, dtype=float))
    P = np.stack([x.ravel(), y.ravel(), np.sin(0.7 * x.ravel())], 1) + rng.uniform(-0.2, 0.2, (nx * ny, 3))
    i = (np.arange(ny - 1)[:, None] * nx + np.arange(nx - 1)).ravel()
    T = np.concatenate([np.stack([i, i + 1, i + nx + 1], 1), np.stack([i, i + nx + 1, i + nx], 1)])
    return P.astype(np.float32), T.astype(np.int64)


def _batch(name, band):
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    P, T, _, vofs, tofs = concat_charts([_grid(*s, seed=k) for k, s in enumerate(SIZES[name])], with_uv=False)
    db = DeviceBatch(P, T, vofs, tofs)
    if not band:
        db.desc.band = None
        db.setup()
    return db


def _call(db, kind, iters=1):
    from ultimate_uv_artist_b200 import _lib
    prm = db.params(kind, iters=iters)
    f = getattr(_lib.lib(), "uva_" + kind)
    _lib.check(f(C.byref(db.desc), C.byref(prm), db._stream()), kind)   # db.desc: no scratch for factors
    torch.cuda.synchronize()
    return db.uvs().copy()


@pytest.mark.parametrize("name", sorted(SIZES))
def test_left_out_operators_match(cuda, name):
    a, b = _batch(name, True), _batch(name, False)
    assert np.array_equal(_call(a, "lscm"), _call(b, "lscm"))
    for it in (1, 2):
        assert np.array_equal(_call(a, "arap", it), _call(b, "arap", it)), it
    c = _batch(name, True)   # a factor solve first, then CG
    c.lscm()
    b.U[:b.n].copy_(c.U[:c.n])
    assert np.array_equal(_call(c, "arap", 2), _call(b, "arap", 2))
    c.setup()                # a new set-up leaves them out again
    b.U[:b.n].copy_(c.U[:c.n])
    assert np.array_equal(_call(c, "arap", 2), _call(b, "arap", 2))


def test_left_out_operators_under_capture(cuda):
    from ultimate_uv_artist_b200 import _lib
    a, b = _batch("cta", True), _batch("cta", False)
    start = _call(b, "lscm")
    s = torch.cuda.Stream()
    want = _call(b, "arap", 2)
    g = torch.cuda.CUDAGraph()
    prm = a.params("arap", iters=2)
    with torch.cuda.graph(g, stream=s):
        _lib.check(_lib.lib().uva_arap(C.byref(a.desc), C.byref(prm), C.c_void_p(s.cuda_stream)), "uva_arap")
    for _ in range(2):
        a.U[:a.n].copy_(torch.from_numpy(start))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(a.uvs(), want)
