"""Grids with many more linked cells than a full tank has (0.02 a particle):
two tanks apart, one of them far enough that most cells between are empty.  Up
to 32,768 cells the row numbering visits every cell, beyond it lists the
occupied ones; a tile may hold rows of both tanks; past 65,536 cells and 64 a
particle the default is the 8-byte layout, and the compact one can still be
asked for.  One step against the 8-byte layout at test_gpu_tiles.py's bound
(at most as many rows as particles)."""
import os

import numpy as np
import pytest

from test_gpu_tiles import _flow, _params

pytestmark = pytest.mark.gpu

TUNE = {"stage_threads": 256, "ppe_threads": 1024, "ppe_stored_weights": 1, "ppe_pipelined": 0, "ppe_compact": 1}


def _apart(cells):
    """Two tanks in a grid of about `cells` linked cells."""
    edge = 0.04 * cells ** (1 / 3) - 0.2
    a, b = _flow((14, 8, 13), (9, 6, 10), 0.01), _flow((13, 9, 11), (10, 5, 8), 0.01, speed=0.6)
    parts = []
    for lo, hi in ((0, 2), (2, 3), (3, None)):  # dummies, walls, fluid of both
        for k, (pos, vel, nb2, nb1) in enumerate((a, b)):
            at = (0, 0, nb2, nb2 + nb1, None)
            s = slice(at[lo], at[hi] if hi else None)
            parts.append((pos[s] + np.float32(k * edge), vel[s]))
    return (np.concatenate([p for p, _ in parts]), np.concatenate([v for _, v in parts]), a[2] + b[2], a[3] + b[3])


def _close(a, b, n):
    top = np.abs(b["press"]).max()
    tol = 5e-7 * np.sqrt(n) + 1e-6
    assert top > 0 and np.abs(a["press"].astype(np.float64) - b["press"]).max() <= tol * top
    assert np.abs(a["vel"].astype(np.float64) - b["vel"]).max() <= 32 * 5e-4 / 1000.0 / 0.01 * tol * top + 1e-6


@pytest.mark.parametrize("cells,learned,arith", [(20000, False, "fast"), (45000, False, "fast"), (150000, True, "fast"),
                                                 (150000, False, "exact"), (1500000, False, "fast")])
def test_two_tanks_apart(capi, cells, learned, arith):
    from mps_solvers_b200 import precond_weights
    pos, vel, nb2, nb1 = _apart(cells)
    prefers = cells <= 64 * len(pos)
    assert prefers == (cells < 1000000)
    opt = dict(method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT,
               precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL)
    out = []
    for layout in (0, -1):
        with capi.Simulation.from_arrays(_params(capi, 0.01, 5e-4), pos, nb2, nb1, vel, ppe_layout=layout, **opt) as s:
            g = s.scalars()["ncells"] / (4 if arith == "fast" else 1)
            assert 0.7 * cells < g < 1.4 * cells
            assert (s.scalars()["ppe_escaped"] >= 0) == (prefers and layout == 0)
            if layout == 0 and not prefers:
                s.apply_tuning(TUNE)
            if learned:
                s.set_precond_params(precond_weights.load())
            for _ in range(2):
                st = s.step(1)
                assert st.status == 0 and st.cg_relres <= 1e-8
                out.append((s.state(capi.ORDER_BY_ID), s.ppe_stencil()))
            assert (s.scalars()["ppe_escaped"] >= 0) == (layout == 0)
    for (a, ea), (b, eb) in zip(out[:2], out[2:]):
        _close(a, b, len(pos))
    for f in ("row_start", "cols", "weights"):  # of the first step, from the same state
        assert np.array_equal(out[0][1][f], out[2][1][f]), f


def test_viscosity_of_two_tanks_apart(capi):
    pos, vel, nb2, nb1 = _apart(100000)
    p = _params(capi, 0.01, 5e-4)
    p.niu = 1e-2
    out = []
    for layout in (0, -1):
        with capi.Simulation.from_arrays(p, pos, nb2, nb1, vel, method=capi.METHOD_SEMI_IMPLICIT, visc_implicit=1,
                                         arith=capi.ARITH_FAST, ppe_layout=layout) as s:
            assert s.step(1).status == 0
            out.append(s.state(capi.ORDER_BY_ID))
    a, b = out
    assert np.abs(a["pos"] - b["pos"]).max() / np.abs(b["pos"]).max() < 1e-6
    assert np.abs(a["vel"] - b["vel"]).max() / np.abs(b["vel"]).max() < 1e-3


@pytest.mark.parametrize("learned", [False, True])
def test_batch_of_tanks_apart(capi, tmp_path, learned):
    from mps_solvers_b200 import precond_weights, scene
    dirs = []
    for k, cells in enumerate((60000, 30000)):
        dirs.append(str(tmp_path / str(k)))
        os.makedirs(dirs[-1])
        pos, vel, nb2, nb1 = _apart(cells)
        prm = scene.Params(dim=3, dp=0.01, r0=2.1, rlap=4.0, cs=20.0, dt_max=5e-4, tt=1.0, max_dis=0.01)
        scene.write_input_dat(os.path.join(dirs[-1], "input.dat"), prm)
        scene.write_geo_dat(os.path.join(dirs[-1], "GEO.dat"), pos, nb2, nb1, vel)
    out = []
    for layout in (0, -1):
        with capi.Simulation.batch(dirs, method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST, ppe_layout=layout,
                                   precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL) as s:
            if learned:
                s.set_precond_params(precond_weights.load())
            assert s.step(1).status == 0
            assert (s.scalars()["ppe_escaped"] >= 0) == (layout == 0)
            out.append(s.state(capi.ORDER_BY_ID))
    _close(*out, len(out[0]["press"]))
