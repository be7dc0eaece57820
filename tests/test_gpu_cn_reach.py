"""Crank-Nicolson viscosity: pairs that come within rlap while the components
move.  The cells are those of the last sort; the x component's solve moves a
particle of the next cell to 3.88 spacings from one that left its own cell on
the other side, whose cells past the face are 4.02 spacings away.  The y
component couples them (for both: the matrix is symmetric); a second pair the
same along y, for z.  Against the FP64 oracle, which visits all 27 linked
cells, at test_gpu_cn.py's bound; without the coupling the velocities it
changes are off by some 0.2 of the largest one."""
import os

import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu

L0, DT = 0.01, 5e-4


def _case(d):
    from mps_solvers_b200 import scene
    os.makedirs(d)
    # cell faces at -0.01 + 0.04 k; a pair of neighbours for n0, a far corner
    pos = np.array([[0, 0, 0], [0.01, 0, 0], [0.25, 0.13, 0.13],
                    [0.07001, 0.05, 0.05], [0.1105, 0.05, 0.05],
                    [0.17, 0.03001, 0.05], [0.17, 0.0705, 0.05]], np.float32)
    vel = np.zeros((7, 3), np.float32)
    vel[3, 0], vel[4, 0] = -0.02 * L0 / DT, -0.19 * L0 / DT
    vel[5, 1], vel[6, 1] = -0.02 * L0 / DT, -0.19 * L0 / DT
    vel[4, 1] = vel[6, 2] = 1.0
    p = scene.Params(dim=3, dp=L0, r0=2.1, rlap=4.0, cs=20.0, dt_max=DT, tt=1.0, niu=1.0, max_dis=L0)
    scene.write_input_dat(os.path.join(d, "input.dat"), p)
    scene.write_geo_dat(os.path.join(d, "GEO.dat"), pos, 0, 0, vel)
    return d


@pytest.mark.parametrize("layout", [0, -1])
@pytest.mark.parametrize("arith", ["exact", "fast"])
def test_pairs_that_move_into_reach(capi, oracle_mod, tmp_path, layout, arith):
    d = _case(str(tmp_path / "c"))
    orc = oracle_mod.Oracle(d, oracle_mod.SEMI_JACOBI, 64)
    orc.set_cg(True, 1e-12, 100000)
    orc.set_visc_implicit(True)
    assert orc.step(1) == 0
    ref = orc.state()
    ref = ref["vel"][np.argsort(ref["id"])]
    with capi.Simulation(d, method=capi.METHOD_SEMI_IMPLICIT, visc_implicit=1, ppe_layout=layout,
                         arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT) as s:
        st = s.step(1)
        assert st.status == 0 and st.cg_relres <= 1e-8
        vel = s.state(capi.ORDER_BY_ID)["vel"]
    assert ref[3, 1] > 0.1 and ref[5, 2] > 0.1 - 9.81 * DT  # the pairs are coupled
    assert rel_err(vel, ref) < 1e-3
