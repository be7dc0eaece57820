"""A matrix large enough that the tile solver fetches its chunks into L2 ahead
of their loads (ppe_compact.cu: C16_AHEAD_FROM chunks) against the 8-byte
layout; the system and the bounds are test_gpu_tiles.py's."""
import numpy as np
import pytest

from test_gpu_tiles import _flow, _step

pytestmark = pytest.mark.gpu


def test_fetched_tiles_match_8_byte_layout(capi):
    args = _flow((101, 91, 107), (87, 88, 97), 0.01)
    a, ea, rows, ita = _step(capi, args, ppe_layout=0, arith=capi.ARITH_FAST)
    b, eb, _, itb = _step(capi, args, ppe_layout=-1, arith=capi.ARITH_FAST)
    # slices of 8 rows hold at least their entries in chunks of 128
    assert len(ea["weights"]) >= 700000 * 128
    assert np.array_equal(ea["weights"], eb["weights"])
    tol = (5e-7 * np.sqrt(rows) + 1e-6) * np.abs(b["press"]).max()
    assert np.abs(a["press"].astype(np.float64) - b["press"]).max() <= tol
    assert abs(ita - itb) <= max(2, itb // 10)
