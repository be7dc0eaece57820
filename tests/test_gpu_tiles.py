"""The compact layout's tiles (mps_solvers_b200/csrc/ppe_compact.cu) against the
8-byte layout, where their rules change: a handful of rows (most blocks of
the solver without a tile, slices partly filled), odd sizes with one tile a
block, and more rows than one tile a block takes (several tiles, the rows'
state in global memory), with diagonal scaling and with the learned form.

One step from the same state.  The pair sets and weights are the same matrix.
Both solves end at |b - A x| <= 1e-8 |b|, so the solutions differ by at most
2e-8 kappa |x| in the 2-norm, kappa ~ 25 for this matrix (its compressibility
term is 3 to 5 % of the diagonal); the largest difference is at most the
2-norm, sqrt(R) rms: 5e-7 sqrt(R) of the largest pressure, and float rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(capi, l0, dt):
    p = capi.mps_params()
    p.dim = 3
    for k, v in dict(rho=1000.0, niu=1e-6, dp=l0, rzero=2.1 * l0, rlap=4.0 * l0, beta=0.97, cs=20.0, cfl=0.2,
                     col_dis=0.8 * l0, col_rate=2.0, dt_max=dt, dt_min=1e-3 * dt, tt=1.0, tout=1e9,
                     max_dis=l0).items():
        setattr(p, k, v)
    return p


def _flow(interior, fluid, l0, speed=0.8):
    """A column of water running into the corner of its tank."""
    from mps_solvers_b200 import scene
    sc = scene.Scene(l0=l0, interior=interior, fluid=[scene.Box(0, 0, 0, *fluid)], jitter=2e-4, seed=3)
    pos, nb2, nb1 = scene.build(sc)
    vel = np.zeros_like(pos)
    f = pos[nb2 + nb1:] / np.float32(l0) - 2 * sc.wall_layers
    vel[nb2 + nb1:, 0] = -speed * (0.25 + 0.75 * f[:, 0] / fluid[0])
    vel[nb2 + nb1:, 2] = -speed * (0.25 + 0.75 * f[:, 2] / fluid[2])
    return pos, vel, nb2, nb1


def _step(capi, scene_args, **opt):
    pos, vel, nb2, nb1 = scene_args
    with capi.Simulation.from_arrays(_params(capi, 0.01, 5e-4), pos, nb2, nb1, vel,
                                     method=capi.METHOD_SEMI_IMPLICIT, **opt) as s:
        if opt.get("precond"):
            from mps_solvers_b200 import precond_weights
            s.set_precond_params(precond_weights.load())
        st = s.step(1)
        assert st.status == 0 and st.cg_relres <= 1e-8
        e = s.ppe_stencil()
        return s.state(capi.ORDER_BY_ID), e, int(s.ppe_snapshot()["is_row"].sum()), st.cg_iters


SCENES = {
    "few rows": ((9, 7, 9), (3, 3, 4)),
    "one tile a block": ((41, 13, 29), (17, 13, 23)),
    "several tiles a block": ((82, 63, 87), (71, 60, 79)),
}


@pytest.mark.parametrize("name,learned,arith", [
    ("few rows", False, "exact"), ("few rows", True, "fast"), ("one tile a block", False, "fast"),
    ("one tile a block", True, "exact"), ("several tiles a block", False, "fast"),
    ("several tiles a block", True, "fast")])
def test_tiles_match_8_byte_layout(capi, name, learned, arith):
    args = _flow(*SCENES[name], 0.01)
    opt = dict(arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT,
               precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL)
    a, ea, rows, ita = _step(capi, args, ppe_layout=0, **opt)
    b, eb, rows_b, itb = _step(capi, args, ppe_layout=-1, **opt)
    assert rows == rows_b
    if name == "several tiles a block":
        assert rows > 148 * 1600
    for f in ("row_start", "cols", "weights"):
        assert np.array_equal(ea[f], eb[f]), f
    top = np.abs(b["press"]).max()
    assert top > 0
    tol = 5e-7 * np.sqrt(rows) + 1e-6
    assert np.abs(a["press"].astype(np.float64) - b["press"]).max() <= tol * top
    # u changes by dt / rho grad p: the pressures' difference over one spacing
    # and 32 neighbours
    assert np.abs(a["vel"].astype(np.float64) - b["vel"]).max() <= 32 * 5e-4 / 1000.0 / 0.01 * tol * top + 1e-6
    assert abs(ita - itb) <= max(2, itb // 10)
