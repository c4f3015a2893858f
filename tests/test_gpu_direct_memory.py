"""Without device memory for the factors a call takes CG, says so and meets its
tolerance; a call of too few iterations for factors asks for no memory."""
import warnings

import numpy as np
import pytest
import torch

from test_gpu_direct import UV_TOL, _grid

pytestmark = pytest.mark.gpu


def test_no_memory_for_factors(cuda, monkeypatch):
    from ultimate_uv_artist_b200 import device
    P, T, _, vofs, tofs = device.concat_charts([_grid(30, 30, seed=1), _grid(9, 9, seed=2)], with_uv=False)
    db = device.DeviceBatch(P, T, vofs, tofs)
    db.lscm()
    start = db.uvs().copy()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        db.arap(iters=4)
    want = db.uvs().copy()
    assert (db.island_status()["cg_iters"] == 0).all()
    asked = []
    empty = torch.empty

    def refuse(*a, **kw):
        if kw.get("dtype") == torch.uint8:
            asked.append(a)
            raise torch.cuda.OutOfMemoryError("no memory")
        return empty(*a, **kw)

    monkeypatch.setattr(device.torch, "empty", refuse)
    db.U[:db.n].copy_(torch.from_numpy(start))
    with pytest.warns(RuntimeWarning, match="memory for the factors of arap"):
        db.arap(iters=4)
    st = db.island_status()
    assert (st["cg_iters"] > 0).all() and (st["resid"] <= 2e-7 * 1.001).all()
    got = db.uvs()
    for a, e in zip(vofs[:-1], vofs[1:]):
        assert np.abs(got[a:e] - want[a:e]).max() <= UV_TOL * np.ptp(want[a:e], 0).max()
    with pytest.warns(RuntimeWarning, match="memory for the factors of lscm"):
        db.lscm()
    assert len(asked) == 2
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        db.arap(iters=2)
    assert len(asked) == 2
