"""The schedule knobs act on CG only, so the autotuner's trials solve every
island by CG, also those that an ordinary call of three iterations solves by
factors; the UVs are as before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_trials_run_cg(cuda):
    from ultimate_uv_artist_b200 import autotune, synth
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    charts = synth.uneven_islands(seed=71, count=40, tmin=60, tmax=3000)
    P, T, _, vofs, tofs = concat_charts([(p, t) for p, t in charts], with_uv=False)
    db = DeviceBatch(P, T, vofs, tofs)
    db.lscm()
    db.arap(iters=3)
    assert (db.island_status()["cg_iters"] == 0).all()
    U0 = db.uvs().copy()
    best, res = autotune.tune(db, use_cache=False)
    assert len(res) == 12 and all(ms > 0 for ms in res.values())
    assert (db.island_status()["cg_iters"] > 0).all()
    torch.cuda.synchronize()
    assert np.array_equal(db.uvs(), U0)
