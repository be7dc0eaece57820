"""The tile layout past its limits (mps_solvers_b200/csrc/ppe_compact.cu): a
column that is not in its tile's list is coded as escaped, and a tile that
does not fit a block's shared memory is done by one warp.  Scenes that get
there have hundreds of thousands of rows of very uneven density, so these
tests build the library with lower limits: tiles that list 320 columns, and
tiles whose columns come from one page of 256 rows, each by one warp.

Rows here have up to 460 entries (rlap = 4.7 spacings).  A tile that holds one
must escape some: in the first build it lists 320 columns; in the second its
own rows, at most ROWS, and 256 more.  ROWS follows from the cut: tiles carry
equal shares of the slices' chunks + 5, a slice has 1 to 29 chunks, so a tile
has at most 34 / 6 of the average slices and one, of 8 rows.

Matrix and results against the 8-byte layout of the same build, as in
test_gpu_tiles.py; its bound on the pressures follows the matrix's
compressibility term, which is (4.7 / 4)^3 times smaller here beside the
diagonal: 8.5e-7 sqrt(R) of the largest.
"""
import importlib.util
import os

import numpy as np
import pytest

from helpers import rel_err
from test_gpu_tiles import _flow, _params

pytestmark = pytest.mark.gpu

BUILDS = {"cols": ["MPS_C16_COLS=320"], "pages": ["MPS_C16_PAGES=1", "MPS_C16_WHOLE=1"]}
SCENE = ((13, 10, 14), (11, 10, 12))


@pytest.fixture(scope="module")
def variants(capi):
    from mps_solvers_b200 import build
    out = {}
    for name, defines in BUILDS.items():
        spec = importlib.util.spec_from_file_location(f"capi_{name}", capi.__file__)
        m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(m)
        m.LIB_PATH = build.build_variant(name, defines)
        out[name] = m
    return out


def _tile_rows(rows, tiles=148):
    return int(8 * (34 / 6 * rows / 8 / tiles + 1))


def _options(m, learned, arith):
    return dict(method=m.METHOD_SEMI_IMPLICIT, arith=m.ARITH_FAST if arith == "fast" else m.ARITH_EXACT,
                precond=m.PRECOND_LEARNED if learned else m.PRECOND_DIAGONAL)


@pytest.mark.parametrize("build,learned,arith", [("cols", False, "fast"), ("cols", True, "exact"),
                                                 ("pages", False, "exact"), ("pages", True, "fast")])
def test_escaped_columns(variants, build, learned, arith):
    from mps_solvers_b200 import precond_weights
    m = variants[build]
    pos, vel, nb2, nb1 = _flow(*SCENE, 0.01)
    p = _params(m, 0.01, 5e-4)
    p.rlap = 4.7 * 0.01
    out = []
    for layout in (0, -1):
        with m.Simulation.from_arrays(p, pos, nb2, nb1, vel, ppe_layout=layout, **_options(m, learned, arith)) as s:
            if learned:
                s.set_precond_params(precond_weights.load())
            st = s.step(1)
            assert st.status == 0 and st.cg_relres <= 1e-8
            out.append((s.state(m.ORDER_BY_ID), s.ppe_stencil(), int(s.ppe_snapshot()["is_row"].sum()), st.cg_iters))
    (a, ea, rows, ita), (b, eb, _, itb) = out
    longest = np.diff(ea["row_start"].astype(np.int64)).max()
    assert _tile_rows(rows) <= 320  # a tile lists its own rows
    assert longest > (320 if build == "cols" else _tile_rows(rows) + 256)
    for f in ("row_start", "cols", "weights"):
        assert np.array_equal(ea[f], eb[f]), f
    top = np.abs(b["press"]).max()
    tol = 8.5e-7 * np.sqrt(rows) + 1e-6
    assert np.abs(a["press"].astype(np.float64) - b["press"]).max() <= tol * top
    assert np.abs(a["vel"].astype(np.float64) - b["vel"]).max() <= 32 * 5e-4 / 1000.0 / 0.01 * tol * top + 1e-6
    assert abs(ita - itb) <= max(2, itb // 10)


@pytest.mark.parametrize("build", ["cols", "pages"])
def test_escaped_columns_of_the_viscosity(variants, build):
    m = variants[build]
    pos, vel, nb2, nb1 = _flow(*SCENE, 0.01)
    p = _params(m, 0.01, 5e-4)
    p.rlap, p.niu = 4.7 * 0.01, 1.0
    out = []
    for layout in (0, -1):
        with m.Simulation.from_arrays(p, pos, nb2, nb1, vel, ppe_layout=layout, visc_implicit=1,
                                      **_options(m, False, "fast")) as s:
            st = s.step(1)
            assert st.status == 0 and st.cg_relres <= 1e-8
            out.append(s.state(m.ORDER_BY_ID))
    a, b = out
    assert np.abs(a["pos"] - b["pos"]).max() / np.abs(b["pos"]).max() < 1e-6
    assert rel_err(a["vel"], b["vel"]) < 1e-3


@pytest.mark.parametrize("build,learned", [("cols", True), ("pages", False), ("pages", True)])
def test_escaped_columns_of_a_batch(variants, tmp_path, build, learned):
    from mps_solvers_b200 import precond_weights, scene
    m = variants[build]
    dirs = []
    for k, (interior, fluid) in enumerate([((9, 7, 9), (3, 3, 4)), SCENE]):
        dirs.append(str(tmp_path / str(k)))
        os.makedirs(dirs[-1])
        pos, vel, nb2, nb1 = _flow(interior, fluid, 0.01)
        prm = scene.Params(dim=3, dp=0.01, r0=2.1, rlap=4.7, cs=20.0, dt_max=5e-4, tt=1.0, max_dis=0.01)
        scene.write_input_dat(os.path.join(dirs[-1], "input.dat"), prm)
        scene.write_geo_dat(os.path.join(dirs[-1], "GEO.dat"), pos, nb2, nb1, vel)
    out = []
    for layout in (0, -1):
        with m.Simulation.batch(dirs, ppe_layout=layout, **_options(m, learned, "fast")) as s:
            if learned:
                s.set_precond_params(precond_weights.load())
            assert s.step(1).status == 0
            infos = [s.scene_info(k) for k in range(2)]
            assert all(i.cg_relres <= 1e-8 for i in infos)
            out.append((s.state(m.ORDER_BY_ID), s.ppe_stencil(), infos))
    (a, ea, ia), (b, eb, _) = out
    if build == "cols":
        assert np.diff(ea["row_start"].astype(np.int64)).max() > 320
    for f in ("row_start", "cols", "weights"):
        assert np.array_equal(ea[f], eb[f]), f
    for i in ia:
        sl = slice(i.id_base, i.id_base + i.np0)
        top = np.abs(b["press"][sl]).max()
        tol = 8.5e-7 * np.sqrt(i.np0 - i.nb2) + 1e-6  # at most as many rows
        assert np.abs(a["press"][sl].astype(np.float64) - b["press"][sl]).max() <= tol * top
