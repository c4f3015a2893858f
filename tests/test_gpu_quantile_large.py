"""The 95 % quantiles of charts around and above the size from which a cluster
of CTAs shares an island (16,384 triangles), alone, among small ones and more of
them than clusters. The anisotropy returned is one of the chart's own and the
weight below and up to it encloses 95 %, to 1e-10, the round-off of sums of
70,000 FP64 terms; the area quantile is that of |log2| and taken back, so its
neighbours to 1e-12 count with it."""
import numpy as np
import pytest

from test_gpu_energy_edges import _strip

pytestmark = pytest.mark.gpu


def _encloses(x, w, v, near=0.0, q=0.95):
    total = w.sum()
    return (w[x < v * (1 - near)].sum() <= (q + 1e-10) * total
            and w[x <= v * (1 + near)].sum() >= (q - 1e-10) * total)


@pytest.mark.parametrize("sizes", [[16383, 16384, 16385], [70001], [3, 65536, 5, 16385, 200], [40] * 50 + [17000] * 40],
                         ids=["edges", "one", "among", "many"])
def test_quality_of_large_charts(cuda, sizes):
    from ultimate_uv_artist_b200 import _lib
    from ultimate_uv_artist_b200.device import DeviceBatch, concat_charts
    from ultimate_uv_artist_b200.engine import param
    rng = np.random.default_rng(len(sizes))
    made = {t: _strip(t, rng) for t in sorted(set(sizes))}
    charts = [made[t] for t in sizes]
    P, T, _, vofs, tofs = concat_charts(charts, with_uv=False)
    U = np.concatenate([p[:, :2].astype(np.float64) + rng.normal(0, 0.02, (len(p), 2)) for p, _ in charts])
    db = DeviceBatch(P, T, vofs, tofs, U=U, semantics=_lib.SEM_PARAM)
    for (p, t), r in zip(charts, param.chart_quality_batch(db)):
        p = p.astype(np.float64)
        w = 0.5 * np.linalg.norm(np.cross(p[t[:, 1]] - p[t[:, 0]], p[t[:, 2]] - p[t[:, 0]]), axis=1)
        assert (r["per_tri_aniso"] == r["aniso_p95"]).any() and _encloses(r["per_tri_aniso"], w, r["aniso_p95"])
        ratio = np.exp2(np.abs(np.log2(np.maximum(r["per_tri_area"], 1e-12))))
        assert _encloses(ratio, w, r["area_p95"], 1e-12)
