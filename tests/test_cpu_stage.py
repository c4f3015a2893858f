"""The parallel staging copy of host arrays (uva_stage) against numpy's
astype: equal types, float64 -> float32, int64 -> int32; empty arrays, one
range, range remainders."""
import ctypes as C

import numpy as np
import pytest

CODE = {np.dtype(np.float32): 0, np.dtype(np.float64): 1, np.dtype(np.int32): 2, np.dtype(np.int64): 3}


@pytest.mark.parametrize("n", [0, 1, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 3 * (1 << 18) + 77])
@pytest.mark.parametrize("pair", [("f4", "f4"), ("f8", "f8"), ("i4", "i4"), ("i8", "i8"), ("f8", "f4"), ("i8", "i4")])
def test_stage_matches_astype(n, pair):
    from ultimate_uv_artist_b200 import _lib
    rng = np.random.default_rng(n)
    s, d = np.dtype(pair[0]), np.dtype(pair[1])
    if s.kind == "f":
        a = (rng.normal(0, 1, n) * 10.0 ** rng.integers(-50, 50, n)).astype(s)
        a[: n // 7 : 3] = np.nan
        a[1 : n // 5 : 4] = -np.inf
    else:
        a = rng.integers(-(1 << 40) if s.itemsize == 8 else -(1 << 30), 1 << 30, n).astype(s)
    out = np.full(n + 1, 7, d)
    rc = _lib.lib().uva_stage(C.c_void_p(a.ctypes.data), CODE[s], C.c_void_p(out.ctypes.data), CODE[d], n)
    with np.errstate(over="ignore"):
        want = a.astype(d)
    assert rc == 0 and out[n] == 7
    assert out[:n].tobytes() == want.tobytes()


def test_stage_refuses_other_pairs():
    from ultimate_uv_artist_b200 import _lib
    a = np.zeros(4)
    p = C.c_void_p(a.ctypes.data)
    for src, dst in ((0, 1), (2, 3), (1, 2), (4, 4), (-1, -1)):
        assert _lib.lib().uva_stage(p, src, p, dst, 4) != 0
    assert _lib.lib().uva_stage(None, 0, p, 0, 4) != 0
    assert _lib.lib().uva_stage(p, 0, p, 0, -1) != 0
