"""Placement against the oracle where many corners pass the filter rows of a
chart and fail on others: combs (several runs per row, the teeth between the
filter rows), plain boxes around the counts of rows that one test covers (8
rows per thread, 32 per warp), and charts whose turns tie. Placements and
occupancy exactly. The row runs, a warp per row, against the masks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _boxes(rects):
    U, T = [], []
    for x0, y0, x1, y1 in rects:
        k = len(U)
        U += [(x0, y0), (x1, y0), (x1, y1), (x0, y1)]
        T += [(k, k + 1, k + 2), (k, k + 2, k + 3)]
    return np.array(U, np.float64), np.array(T, np.int64)


def _comb(w, h, pitch, depth, phase):
    """A spine of height h with teeth of one row in each `pitch` rows."""
    return _boxes([(0, 0, 2, h)] + [(0, y, depth, y + 0.5) for y in np.arange(phase, h - 0.5, pitch)] + [(w - 1, h - 1, w, h)])


CASES = {
    "combs": [_comb(40, 37, 5, 30, p) for p in (1, 2, 3)] * 5 + [_comb(23, 70, 9, 20, 4)] * 6 + [_boxes([(0, 0, 6, 6)])] * 40,
    "heights": [_boxes([(0, 0, 11 + k % 3, h)]) for k, h in enumerate([1, 2, 6, 7, 8, 9, 14, 15, 16, 30, 31, 32, 33, 63, 64, 65] * 4)],
    "ties": [_boxes([(0, 0, 20, 20)])] * 30 + [_boxes([(0, 0, 8, 30), (0, 0, 30, 8)])] * 20,
}


@pytest.mark.parametrize("G", [129, 320, 512])
@pytest.mark.parametrize("name", sorted(CASES))
def test_placement_matches_oracle(name, G):
    from oracle import pack as OP
    from ultimate_uv_artist_b200.engine import pack as EP
    Us, Ts = [U for U, _ in CASES[name]], [T for _, T in CASES[name]]
    dens = np.ones(len(Us))
    box = sum(float(np.prod(U.max(0) - U.min(0))) for U in Us)
    P = EP.Packer(Us, Ts, dens)
    placed = 0
    for f in (0.35, 0.55, 0.75):
        s = f * float(np.sqrt(G * G / box))
        for rot in ([0], [0, 1, 2, 3]):
            ref = OP.attempt(Us, Ts, dens, G, 1, rot, s, "area", (0.0,))
            att = P.attempt(G, 1, rot, s, "area")
            assert (ref is None) == (att is None), (f, rot)
            if ref is not None:
                placed += 1
                assert att.placement == ref[1][0], (f, rot)
                assert att.occupied == int(ref[1][1].sum())
    assert placed
