"""Batches of a few vertices built on the device: the plan's offset arrays are
a few hundred bytes, so an array allocated between the plan's two passes (the
uploaded positions) fits their blocks; they must stay alive until the second
pass has read them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [1, 2, 3, 5])
def test_tiny_batch_plan_equals_the_host_plan(cuda, cells):
    from ultimate_uv_artist_b200 import synth
    from ultimate_uv_artist_b200.engine import gpu
    rng = np.random.default_rng(cells)
    P, T = synth.disk_patch(rng, 2 * cells * cells)
    assert len(P) <= 42
    host = gpu.Batch([(P, T, None)], plan_on="host")
    dev = gpu.Batch([(P, T, None)])
    for name in ("tri4", "tri_edge", "slice_ptr", "slot_col", "slot_edge", "slot_c", "vt_ptr", "vt", "bverts"):
        assert torch.equal(getattr(dev.db, name), getattr(host.db, name)), name
    assert np.isfinite(np.concatenate([u for u in (dev.lscm().cpu().numpy(),)])).all()
