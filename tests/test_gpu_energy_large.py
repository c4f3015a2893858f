"""Energies of triangles whose squared normal overflows FP64 (edges of 1e80):
infinite, as the same formulas in plain FP64 torch say, and not left out."""
import numpy as np
import pytest
import torch

from test_gpu_energy_edges import _reference, _strip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1e70, 1e80])
def test_large_triangles(cuda, kind, scale):
    from ultimate_uv_artist_b200.energy import distortion_energy
    from ultimate_uv_artist_b200.engine import gpu
    rng = np.random.default_rng(3)
    charts = [_strip(t, rng) for t in (3, 40)]
    b = gpu.Batch([(p, t, None) for p, t in charts])
    P = np.concatenate([p for p, _ in charts]).astype(np.float64) * scale
    n0 = len(charts[0][0])
    F = np.concatenate([charts[0][1], charts[1][1] + n0])
    lab = np.repeat([0, 1], [3, 40])
    U = P[:, :2] @ np.array([[1.1, 0.2], [-0.1, 0.9]])
    ref = _reference(P, F, lab, U, 2, kind, False)[0]
    assert bool(torch.isinf(ref).all()) == (scale == 1e80)
    with torch.no_grad():
        e = distortion_energy(b.db, torch.from_numpy(U).to(cuda), torch.from_numpy(P).to(cuda), kind).cpu()
    if scale == 1e80:
        assert torch.equal(e, ref)
    else:
        assert float(((e - ref).abs() / ref).max()) <= 1e-11   # 40 terms of some fifty operations each
