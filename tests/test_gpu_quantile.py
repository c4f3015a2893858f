"""Weighted quantiles (uva_wquantile, the report's and the per-island ones)
against numpy's argsort / cumsum / searchsorted. Weights are small integers,
so every order of summation is exact and the selected values must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy(x, w, q):
    o = np.argsort(x, kind="stable")
    c = np.cumsum(w[o])
    return x[o][min(np.searchsorted(c, q * c[-1]), len(x) - 1)]


@pytest.mark.parametrize("n", [1, 2, 31, 33, 511, 513, 148 * 512 + 1, 300001])
@pytest.mark.parametrize("kind", ["spread", "equal", "signs", "few"])
def test_wquantile_matches_numpy(cuda, n, kind):
    from ultimate_uv_artist_b200.engine import metrics
    rng = np.random.default_rng(n)
    x = {"spread": np.exp(rng.normal(0, 20, n)), "equal": np.full(n, 1.25),
         "signs": rng.normal(0, 1, n) * 10.0 ** rng.integers(-200, 200, n), "few": rng.integers(0, 3, n) * 0.5}[kind]
    w = rng.integers(0, 5, n).astype(np.float64)
    w[rng.integers(0, n)] = 3.0
    for q in (0.0, 0.5, 0.95, 1.0):
        got = metrics._wquantile(x, w, q)
        keep = w > 0          # numpy's q = 0 may land on a value of no weight
        assert got == _numpy(x[keep], w[keep], q), (n, kind, q)


def test_wquantile_of_nothing(cuda):
    from ultimate_uv_artist_b200.engine import metrics
    assert np.isnan(metrics._wquantile(np.ones(40), np.zeros(40), 0.5))
    assert np.isnan(metrics._wquantile(np.zeros(0), np.zeros(0), 0.5))


@pytest.mark.parametrize("order", ["runs", "interleaved", "random"])
def test_report_island_sums_for_any_label_order(cuda, order):
    """The report's per-island sums fold runs of equal labels along a warp;
    labels may come in any order. Permuting the faces (with their labels)
    changes no term of the report beyond round-off (1e-12 relative: sums of
    3,000 positive FP64 terms)."""
    from ultimate_uv_artist_b200.engine import metrics
    rng = np.random.default_rng(5)
    V = rng.normal(0, 1, (900, 3))
    UV = V[:, :2] * 0.3 + rng.normal(0, 0.01, (900, 2))
    F = rng.integers(0, 900, (3001, 3))
    F[:, 1] = (F[:, 0] + 1 + F[:, 1] % 400) % 900
    F[:, 2] = (F[:, 0] + 500 + F[:, 2] % 300) % 900
    isl = np.sort(rng.integers(0, 7, len(F)))
    ref = metrics.distortion_report(V, F, UV, isl)
    p = {"runs": np.arange(len(F)), "interleaved": np.argsort(np.arange(len(F)) % 31, kind="stable"),
         "random": rng.permutation(len(F))}[order]
    got = metrics.distortion_report(V, F[p], UV, isl[p])
    assert set(got) == set(ref)
    for k, v in ref.items():
        assert got[k] == pytest.approx(v, rel=1e-12), k
