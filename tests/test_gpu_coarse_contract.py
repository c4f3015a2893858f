"""Coarse operators that the set-up left out (islands with a factor) and that
no solve has built: CG must not read them (they hold NaN here), and the
no-allocation entry point must leave the batch's arrays alone. Solved to the
call's tolerance all the same, which the FP64 residual of the status says; with
the operators built by uva_batch_coarse, the iterations of uva_arap."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_coarse_left import _batch

pytestmark = pytest.mark.gpu


def _start(name):
    """A batch after its set-up and LSCM by factors, operators unbuilt."""
    db = _batch(name, True)
    db.coarse_a.fill_(float("nan"))
    db.coarse_l.fill_(float("nan"))
    db.setup()
    db.lscm()
    return db


def _status(db, raw=None):
    st = db.island_status()
    return st if raw is None else raw[:db.nc].cpu().numpy().view(st.dtype).reshape(-1)


def _solved(st, prm):
    assert (st["flags"] == 0).all() and (st["resid"] <= prm.tol).all()


@pytest.mark.parametrize("name", ["small", "cta", "global"])
@pytest.mark.parametrize("kind", ["arap", "lscm"])
def test_solve_without_coarse_work(cuda, name, kind):
    from ultimate_uv_artist_b200 import _lib
    db = _start(name)
    prm = db.params(kind, iters=2)
    desc = _lib.BatchDesc.from_buffer_copy(db.desc)
    desc.coarse_work = None
    f = getattr(_lib.lib(), "uva_" + kind)
    _lib.check(f(C.byref(desc), C.byref(prm), db._stream()), kind)
    torch.cuda.synchronize()
    assert np.isfinite(db.uvs()).all()
    _solved(_status(db), prm)
    assert _lib.lib().uva_batch_coarse(C.byref(desc), db._stream()) == _lib.UVA_E_ARG


@pytest.mark.parametrize("name", ["small", "cta", "global"])
def test_noalloc_leaves_the_batch_alone(cuda, name):
    from ultimate_uv_artist_b200 import _lib
    L = _lib.lib()
    db = _start(name)
    U0 = db.U.clone()
    keep = {k: getattr(db, k).clone() for k in ("coarse_a", "coarse_l", "coarse_work", "band", "x64", "b64", "rc")}
    prm = db.params("arap", iters=3)
    status = torch.zeros_like(db.status)
    desc = _lib.BatchDesc.from_buffer_copy(db.desc)
    desc.status = status.data_ptr()
    _lib.check(L.uva_arap_noalloc(C.byref(desc), C.byref(prm), db._stream()), "uva_arap_noalloc")
    torch.cuda.synchronize()
    for k, v in keep.items():
        now = getattr(db, k)
        assert torch.equal(now.view(torch.uint8), v.view(torch.uint8)), k
    assert np.isfinite(db.uvs()).all()
    _solved(_status(db, status), prm)
    # with the operators: the iterations and the UVs of uva_arap without factors
    _lib.check(L.uva_batch_coarse(C.byref(db.desc), db._stream()), "uva_batch_coarse")
    db.U.copy_(U0)
    _lib.check(L.uva_arap(C.byref(db.desc), C.byref(prm), db._stream()), "uva_arap")
    want, st = db.uvs().copy(), _status(db)
    db.U.copy_(U0)
    _lib.check(L.uva_arap_noalloc(C.byref(desc), C.byref(prm), db._stream()), "uva_arap_noalloc")
    torch.cuda.synchronize()
    assert np.array_equal(db.uvs(), want)
    assert np.array_equal(_status(db, status)["cg_iters"], st["cg_iters"])
