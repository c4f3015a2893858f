"""The energy kernels at the edges of their blocks and warps: batches of one
triangle up to a block and its remainder, and many small islands inside one
warp, against plain FP64 torch autograd. Tolerance: each value is a sum of at
most a dozen terms of some fifty FP64 operations, below 1e-13 of the largest;
1e-11 is asked for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-11


def _strip(t, rng):
    """A strip of t triangles (t + 2 vertices) with jittered corners."""
    k = np.arange(t + 2)
    P = np.stack([0.5 * k, (k % 2).astype(float), 0.0 * k], 1) + rng.uniform(-0.15, 0.15, (t + 2, 3))
    i = np.arange(t)
    T = np.where((i % 2 == 0)[:, None], np.stack([i, i + 2, i + 1], 1), np.stack([i, i + 1, i + 2], 1))
    return P.astype(np.float32), T.astype(np.int64)


def _reference(P, F, lab, U, nc, kind, wrt_p):
    P = torch.from_numpy(P.astype(np.float64)).requires_grad_(True)
    U = torch.from_numpy(U).requires_grad_(True)
    F, lab = torch.from_numpy(F), torch.from_numpy(lab)
    e1, e2 = P[F[:, 1]] - P[F[:, 0]], P[F[:, 2]] - P[F[:, 0]]
    x1 = e1.norm(dim=1)
    nn = torch.linalg.cross(e1, e2).norm(dim=1)
    x2, y2 = (e1 * e2).sum(1) / x1, nn / x1
    a = (U[F[:, 1]] - U[F[:, 0]]) / x1[:, None]
    b = (U[F[:, 2]] - U[F[:, 0]] - a * x2[:, None]) / y2[:, None]
    fro = (a * a).sum(1) + (b * b).sum(1)
    det = a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]
    f = fro - 2 * torch.hypot(a[:, 0] + b[:, 1], a[:, 1] - b[:, 0]) + 2 if kind == 0 else fro + fro / det ** 2 - 4
    e = torch.zeros(nc, dtype=torch.float64).index_add(0, lab, 0.5 * nn * f)
    g = torch.linspace(0.5, 1.5, nc, dtype=torch.float64)
    return [e.detach()] + list(torch.autograd.grad((e * g).sum(), (U, P) if wrt_p else (U,)))


@pytest.mark.parametrize("sizes", [[1], [31], [32], [33], [127], [128], [129], [1, 1, 2, 5, 30, 1, 40, 200, 3], [3] * 90],
                         ids=str)
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("wrt_p", [False, True])
def test_energy_and_gradients(cuda, sizes, kind, wrt_p):
    from ultimate_uv_artist_b200.energy import distortion_energy
    from ultimate_uv_artist_b200.engine import gpu
    rng = np.random.default_rng(len(sizes) + sizes[0])
    charts = [_strip(t, rng) for t in sizes]
    b = gpu.Batch([(p, t, None) for p, t in charts])
    P = np.concatenate([p for p, _ in charts])
    ofs = np.cumsum([0] + [len(p) for p, _ in charts])
    F = np.concatenate([t + o for (_, t), o in zip(charts, ofs)])
    lab = np.repeat(np.arange(len(sizes)), sizes)
    U = P[:, :2].astype(np.float64) @ np.array([[1.1, 0.2], [-0.1, 0.9]])
    ref = _reference(P, F, lab, U, len(sizes), kind, wrt_p)
    Ut = torch.from_numpy(U).to(cuda).requires_grad_(True)
    Pt = b.db.P[:b.n].clone().requires_grad_(wrt_p)
    e = distortion_energy(b.db, Ut, Pt, kind)
    g = torch.linspace(0.5, 1.5, len(sizes), dtype=torch.float64, device=cuda)
    got = [e.detach()] + list(torch.autograd.grad((e * g).sum(), (Ut, Pt) if wrt_p else (Ut,)))
    for x, y in zip(got, ref):
        assert float((x.cpu() - y).abs().max()) <= TOL * max(float(y.abs().max()), 1.0)
