"""A batch in which every particle is a row: scenes of nine fluid particles
without walls or dummies, beta = 0.  Each scene's rows start at a multiple of
8, so the row numbers run past the particle count; the batch's matrix, its
learned preconditioner and its results have room for them.  Against the same
scenes alone in the 8-byte layout, one step, at test_gpu_batch_tiles.py's
bounds."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _write(d, k):
    from mps_solvers_b200 import scene
    os.makedirs(d)
    rng = np.random.default_rng(k)
    # a ring of nine shrinking towards its middle: equal densities that all rise, so every pressure is positive
    t = 2 * np.pi * np.arange(9) / 9
    ring = np.stack([np.cos(t), np.sin(t), 0 * t], 1) * 0.01 / (2 * np.sin(np.pi / 9))
    pos = (ring + 1e-6 * (rng.random((9, 3)) - 0.5)).astype(np.float32)
    vel = (-40.0 * ring).astype(np.float32)
    # max_dis widens the grid to the three cells an axis needs
    p = scene.Params(dim=3, dp=0.01, r0=2.1, rlap=4.0, cs=20.0, dt_max=5e-4, tt=1.0, beta=0.0, max_dis=0.1)
    scene.write_input_dat(os.path.join(d, "input.dat"), p)
    scene.write_geo_dat(os.path.join(d, "GEO.dat"), pos, 0, 0, vel)


@pytest.mark.parametrize("scenes,learned,arith", [(2, False, "fast"), (5, True, "exact"), (60, False, "exact"),
                                                  (60, True, "fast")])
def test_batch_of_rows_only(capi, tmp_path, scenes, learned, arith):
    from mps_solvers_b200 import precond_weights
    dirs = [str(tmp_path / str(k)) for k in range(scenes)]
    for k, d in enumerate(dirs):
        _write(d, k)
    opt = dict(method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT,
               precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL)
    with capi.Simulation.batch(dirs, **opt) as b:
        if learned:
            b.set_precond_params(precond_weights.load())
        assert b.step(1).status == 0
        assert b.scalars()["ppe_escaped"] >= 0  # the compact layout
        st = b.ppe_stencil()
        assert (np.diff(st["row_start"].astype(np.int64)) == 8).all()  # all nine rows of a scene couple
        got = b.state(capi.ORDER_BY_ID)
    for k in {0, 1, scenes // 2, scenes - 1}:
        with capi.Simulation(dirs[k], ppe_layout=-1, **opt) as s:
            if learned:
                s.set_precond_params(precond_weights.load())
            assert s.step(1).status == 0
            ref = s.state(capi.ORDER_BY_ID)
        sl = slice(9 * k, 9 * k + 9)
        top = np.abs(ref["press"]).max()
        assert top > 0
        tol = 5e-7 * 3 + 1e-6  # sqrt(9) rows
        assert np.abs(got["press"][sl].astype(np.float64) - ref["press"]).max() <= tol * top, k
        assert np.abs(got["vel"][sl].astype(np.float64) - ref["vel"]).max() <= 32 * 5e-4 / 1000.0 / 0.01 * tol * top + 1e-6
