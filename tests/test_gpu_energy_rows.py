"""Energies of islands that end inside the last warp of a large batch, where a
thread of the forward pass takes several rows of 32 triangles and some lanes of
the last warp take one row less: every island's value against plain FP64 torch.
Tolerance: an island sums at most 1,000 non-negative terms of some fifty FP64
operations each, within 1e-12 of its value; 1e-11 is asked for."""
import numpy as np
import pytest
import torch

from test_gpu_energy_edges import _reference, _strip

pytestmark = pytest.mark.gpu
TOL = 1e-11
ROW = 148 * 1024   # triangles from which a thread takes one more row


@pytest.mark.parametrize("rows", [2, 8])
@pytest.mark.parametrize("rem,tail", [(1, [25]), (5, [31]), (12, [2, 3, 27]), (17, [1, 2, 3, 20]), (30, [7]), (31, [1] * 31)],
                         ids=str)
@pytest.mark.parametrize("kind", [0, 1])
def test_islands_in_the_last_rows(cuda, rows, rem, tail, kind):
    from ultimate_uv_artist_b200.energy import distortion_energy
    from ultimate_uv_artist_b200.engine import gpu
    rng = np.random.default_rng(rows + rem)
    strips = {1000: _strip(1000, rng)}
    sizes = [1000] * (rows * ROW // 1000 + 1)
    # the last warp has one full row and rem triangles of the next
    sizes += [32 * rows + (32 + rem - sum(sizes) - sum(tail)) % (32 * rows)] + tail
    for t in sizes:
        strips.setdefault(t, _strip(t, rng))
    charts = [strips[t] for t in sizes]
    assert sum(sizes) % (32 * rows) == (32 + rem) % (32 * rows) and min(8, sum(sizes) // ROW) == rows
    b = gpu.Batch([(p, t, None) for p, t in charts])
    P = np.concatenate([p for p, _ in charts])
    ofs = np.cumsum([0] + [len(p) for p, _ in charts])
    F = np.concatenate([t + o for (_, t), o in zip(charts, ofs)])
    lab = np.repeat(np.arange(len(sizes)), sizes)
    U = P[:, :2].astype(np.float64) @ np.array([[1.1, 0.2], [-0.1, 0.9]])
    ref = _reference(P, F, lab, U, len(sizes), kind, False)[0]
    with torch.no_grad():
        e = distortion_energy(b.db, torch.from_numpy(U).to(cuda), b.db.P[:b.n], kind).cpu()
    assert float(((e - ref).abs() / ref).max()) <= TOL
