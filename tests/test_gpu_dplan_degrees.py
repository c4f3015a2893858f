"""Row order of the device plan on islands whose vertices have fewer than,
exactly and more than eight neighbours (the walk takes four vertices of up to
eight neighbours at once, a wider one by itself) against the host plan,
element for element. Sizes around 8,192 vertices, where the walk's state
moves to global memory."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fans(degree, count):
    """`count` closed fans in a row, neighbours joined through a rim vertex."""
    P, T = [], []
    prev = None
    for k in range(count):
        c = len(P)
        P.append((3.0 * k, 0.0, 0.0))
        ang = 2 * np.pi * np.arange(degree) / degree
        P += [(3.0 * k + np.cos(a), np.sin(a), 0.1 * j) for j, a in enumerate(ang)]
        T += [(c, c + 1 + j, c + 1 + (j + 1) % degree) for j in range(degree)]
        if prev is not None:
            T.append((prev + 1, c + 1 + degree // 2, c + 2 + degree // 2))
        prev = c
    return np.array(P, np.float32), np.array(T, np.int64)


def _grid(w, h):
    x, y = np.meshgrid(np.arange(w), np.arange(h))
    P = np.stack([x.ravel(), y.ravel(), 0.1 * np.sin(x.ravel())], 1).astype(np.float32)
    i = (y[:-1, :-1] * w + x[:-1, :-1]).ravel()
    return P, np.concatenate([np.stack([i, i + 1, i + w + 1], 1), np.stack([i, i + w + 1, i + w], 1)]).astype(np.int64)


@pytest.mark.parametrize("charts", [
    [(d, c) for d in (6, 7, 8, 9) for c in (40, 250)],
    [(d, 30) for d in (31, 32, 33, 64, 65)] + [(300, 5)],
    ["8191", "8192", "8193"],
], ids=["near-eight", "wide", "state"])
def test_row_order_matches_host(cuda, charts):
    from ultimate_uv_artist_b200.device import DevicePlan, Plan, concat_charts
    if charts[0] == "8191":
        P, T = _grid(64, 128)   # 8,192 vertices
        keep = T[(T != 8191).all(1)]
        items = [(P[:8191], keep), (P, T),
                 (np.concatenate([P, [[70, 0, 0]]]).astype(np.float32), np.concatenate([T, [[63, 127, 8192]]]))]
    else:
        items = [_fans(d, c) for d, c in charts]
    _, Tc, _, vofs, tofs = concat_charts(items, with_uv=False, with_t=False)
    host = Plan(None, vofs, tofs, chart_tris=Tc[:2])
    dev = DevicePlan(Tc[:2], vofs, tofs, device=torch.device("cuda", 0))
    assert (np.asarray(host.agg_rows) > 0).any()
    for k in ("row_vert", "vert_row"):
        a = np.asarray(getattr(host, k)).reshape(-1)
        assert np.array_equal(a, getattr(dev, k).cpu().numpy().reshape(-1)[:a.size]), k
