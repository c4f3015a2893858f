"""The pair filter and the tiled gutter at the places where they could differ
from the reference's full evaluation, bit for bit against the oracle: triangle
soups with shared vertices, collinear edges, touching corners, slivers,
negative and far coordinates; atlas sizes around the tiles' and words' edges,
gaps around the first radius and beyond the largest."""
import numpy as np
import pytest

from oracle import validate as OV

pytestmark = pytest.mark.gpu


def _soup(kind, rng, m):
    """UVs (n, 2) float32 and faces of m triangles."""
    if kind == "random":
        c = rng.uniform(0.1, 0.9, (m, 1, 2))
        return (c + rng.normal(0, 0.02, (m, 3, 2))).reshape(-1, 2), np.arange(3 * m).reshape(-1, 3)
    if kind == "shared":          # few vertices, so most pairs share one or two
        n = m // 3
        return rng.uniform(0, 1, (n, 2)), rng.integers(0, n, (m, 3))
    if kind == "lattice":         # collinear edges, touching corners, coincident triangles
        return (rng.integers(0, 24, (3 * m, 2)) / 32.0 + 0.1), np.arange(3 * m).reshape(-1, 3)
    if kind == "slivers":
        c = rng.uniform(0.1, 0.9, (m, 1, 2))
        d = rng.normal(0, 1, (m, 1, 2)) * 0.05
        t = np.array([0.0, 1.0, 0.37])[None, :, None]
        w = rng.uniform(-1, 1, (m, 3, 2)) * 10.0 ** rng.uniform(-9, -4, (m, 1, 1))
        return (c + t * d + w).reshape(-1, 2), np.arange(3 * m).reshape(-1, 3)
    U, F = _soup("random", rng, m)    # "far": outside the unit square, some beyond 1e6
    U = U * 3 - 1
    U[rng.integers(0, len(U), m // 20)] *= 3e7
    return U, F


@pytest.mark.parametrize("kind", ["random", "shared", "lattice", "slivers", "far"])
@pytest.mark.parametrize("m", [40, 700, 4000])
def test_overlap_flags_bit_exact(cuda, kind, m):
    from ultimate_uv_artist_b200.engine import validate as GV
    rng = np.random.default_rng(m + len(kind))
    U, F = _soup(kind, rng, m)
    U = U.astype(np.float32)
    V = rng.normal(0, 1, (len(U), 3))
    dv = GV.DeviceValidation(V, F.astype(np.int32), U).run()
    fl = dv.flags()
    skip = (fl & 4) != 0
    for strict, bit in ((False, 16), (True, 32)):
        want, _ = OV.overlaps_c(U.astype(np.float64), F, skip, 16, strict=strict)
        assert np.array_equal((fl & bit) != 0, np.asarray(want) != 0), (kind, strict)


@pytest.mark.parametrize("res", [33, 63, 64, 65, 128, 130, 200, 257])
@pytest.mark.parametrize("gap", [1, 3, 15, 17, 40, 90])
def test_gutter_matches_the_oracle(cuda, res, gap):
    """Two rectangles, a sliver and a dot, a stated number of texels apart."""
    from ultimate_uv_artist_b200.engine import metrics
    w = max((res - gap) // 3, 2)
    quad = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], float)
    parts = [quad * [w, res - 3] + [1, 1], quad * [w, max(res // 3, 2)] + [1 + w + gap, 2],
             quad * [w, 2] + [1 + w + gap, res - 4], quad * [1, 1] + [min(1 + w + gap, res - 2), res // 2]]
    uv = np.concatenate(parts) / res + 1e-4
    F = np.concatenate([np.array([[0, 1, 2], [0, 2, 3]]) + 4 * k for k in range(4)])
    isl = np.repeat(np.arange(4), 2)
    g, img = metrics.min_gutter(uv, F, isl, res)
    want, wimg = OV.min_gutter(uv, F, isl, res)
    assert np.array_equal(img, wimg)
    assert g == want or (np.isnan(g) and np.isnan(want))


@pytest.mark.parametrize("res", [64, 100, 300])
def test_gutter_of_scattered_islands(cuda, res):
    """Random small triangles, each its own island: ties and touching labels."""
    from ultimate_uv_artist_b200.engine import metrics
    rng = np.random.default_rng(res)
    for count in (2, 5, 30):
        c = rng.uniform(0.02, 0.98, (count, 1, 2))
        uv = (c + rng.normal(0, 1.5 / res, (count, 3, 2))).reshape(-1, 2)
        F = np.arange(3 * count).reshape(-1, 3)
        g, img = metrics.min_gutter(uv, F, np.arange(count), res)
        want, wimg = OV.min_gutter(uv, F, np.arange(count), res)
        assert np.array_equal(img, wimg) and (g == want or (np.isnan(g) and np.isnan(want)))
