"""A batch's tiles (mps_solvers_b200/csrc/ppe_compact.cu) against the batch
solver of the 8-byte layout: scenes of a handful of rows beside larger ones
(their first rows at multiples of 8, gaps between them, tiles cut by scene),
and more scenes than the solver has blocks (several tiny tiles a block).
One step from the same state; bounds as in test_gpu_tiles.py, per scene."""
import os

import numpy as np
import pytest

from test_gpu_tiles import _flow

pytestmark = pytest.mark.gpu

SETS = {
    "uneven": [((9, 7, 9), (3, 3, 4)), ((41, 13, 29), (17, 13, 23)), ((14, 6, 12), (5, 4, 8)), ((30, 11, 25), (13, 10, 19))],
    "one": [((23, 9, 17), (11, 7, 13))],
    "many": [((9, 7, 9 + k % 3), (3 + k % 4, 3, 4 + k % 5)) for k in range(160)],
}


@pytest.mark.parametrize("name,learned,arith", [("uneven", False, "fast"), ("uneven", True, "fast"),
                                                ("uneven", True, "exact"), ("one", False, "exact"),
                                                ("many", False, "fast"), ("many", True, "fast")])
def test_batch_tiles_match_8_byte_layout(capi, tmp_path, name, learned, arith):
    from mps_solvers_b200 import precond_weights, scene
    dirs = []
    for k, (interior, fluid) in enumerate(SETS[name]):
        d = str(tmp_path / str(k))
        os.makedirs(d)
        pos, vel, nb2, nb1 = _flow(interior, fluid, 0.01, speed=0.6 + 0.01 * (k % 7))
        p = scene.Params(dim=3, dp=0.01, r0=2.1, rlap=4.0, cs=20.0, dt_max=5e-4, tt=1.0, max_dis=0.01)
        scene.write_input_dat(os.path.join(d, "input.dat"), p)
        scene.write_geo_dat(os.path.join(d, "GEO.dat"), pos, nb2, nb1, vel)
        dirs.append(d)
    opt = dict(method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT,
               precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL)
    out = []
    for layout in (0, -1):
        with capi.Simulation.batch(dirs, accel=[(0.5 * (k % 3), 1.0) for k in range(len(dirs))], ppe_layout=layout,
                                   **opt) as b:
            if learned:
                b.set_precond_params(precond_weights.load())
            st = b.step(1)
            assert st.status == 0
            infos = [b.scene_info(s) for s in range(len(dirs))]
            out.append((b.state(capi.ORDER_BY_ID), infos))
    (a, ia), (r, ir) = out
    for s in range(len(dirs)):
        assert ia[s].cg_relres <= 1e-8 and ir[s].cg_relres <= 1e-8
        assert abs(ia[s].cg_iters - ir[s].cg_iters) <= max(2, ir[s].cg_iters // 10)
        sl = slice(ia[s].id_base, ia[s].id_base + ia[s].np0)
        top = np.abs(r["press"][sl]).max()
        tol = 5e-7 * np.sqrt(ia[s].np0 - ia[s].nb2) + 1e-6  # at most as many rows
        assert np.abs(a["press"][sl].astype(np.float64) - r["press"][sl]).max() <= tol * top, s
        assert np.abs(a["vel"][sl].astype(np.float64) - r["vel"][sl]).max() <= 32 * 5e-4 / 1000.0 / 0.01 * tol * top + 1e-6
