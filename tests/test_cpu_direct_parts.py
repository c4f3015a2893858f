"""Scratch parts of the direct solver (device.direct_parts): a CTA whose first
island is above the size limit takes islands of the queue after it, so its
part holds the largest of those."""
import numpy as np
import pytest

from ultimate_uv_artist_b200 import _lib
from ultimate_uv_artist_b200.device import direct_parts


@pytest.mark.parametrize("large", [0, 1, 3, 8, 12])
@pytest.mark.parametrize("small", [0, 5, 8, 30])
def test_parts_after_too_large_islands(large, small):
    slots = 8
    rng = np.random.default_rng(large + 100 * small)
    nv = np.concatenate([rng.integers(_lib.DIRECT_MAX_N + 1, 90000, large), rng.integers(3, _lib.DIRECT_MAX_N + 1, small)])
    rng.shuffle(nv)
    order = np.sort(nv)[::-1]
    parts = np.diff(direct_parts(nv, slots), axis=1)
    assert parts.shape == (2, slots)
    later = [v for v in order[slots:] if v <= _lib.DIRECT_MAX_N]
    for j in range(slots):
        takes = [v for v in order[j:j + 1] if v <= _lib.DIRECT_MAX_N] + later   # its first island, then the queue
        own = np.diff(direct_parts([max(takes)], 1), axis=1)[:, 0] if takes and j < len(order) else np.zeros(2)
        assert (parts[:, j] >= own).all(), j
