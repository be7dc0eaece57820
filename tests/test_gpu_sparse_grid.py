"""Grids with many more linked cells than particles (one particle far from
the others): past 65,536 cells and 4 a particle the default is the 8-byte
layout; the compact one can still be asked for, and both give the same step."""
import numpy as np
import pytest

from test_gpu_tiles import _flow, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,compact", [(0.5, True), (30.0, False)])
def test_layout_by_cells(capi, cells, compact):
    pos, vel, nb2, nb1 = _flow((14, 8, 13), (9, 6, 10), 0.01)
    edge = 0.04 * (cells * (len(pos) + 1)) ** (1 / 3)
    assert cells < 4 or cells * len(pos) > 65536
    pos = np.concatenate([pos.min(0)[None] + np.float32(edge), pos]).astype(np.float32)  # a dummy
    vel = np.concatenate([np.zeros((1, 3), np.float32), vel])
    args = (_params(capi, 0.01, 5e-4), pos, nb2 + 1, nb1, vel)
    opt = dict(method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST)
    out = []
    for layout in (0, -1):
        with capi.Simulation.from_arrays(*args, ppe_layout=layout, **opt) as s:
            assert s.step(1).status == 0
            assert (s.scalars()["ppe_escaped"] >= 0) == (compact and layout == 0)
            a = s.state(capi.ORDER_BY_ID)
            if layout == -1 or not compact:
                s.apply_tuning({"stage_threads": 256, "ppe_threads": 1024, "ppe_stored_weights": 1,
                                "ppe_pipelined": 0, "ppe_compact": 1})
            assert s.step(1).status == 0
            assert s.scalars()["ppe_escaped"] >= 0
            out.append((a, s.state(capi.ORDER_BY_ID)))
    tol = 5e-7 * np.sqrt(len(pos)) + 1e-6  # test_gpu_tiles.py's bound, at most as many rows
    for a, b in zip(*out):
        top = np.abs(b["press"]).max()
        assert top > 0 and np.abs(a["press"].astype(np.float64) - b["press"]).max() <= tol * top
