"""The Crank-Nicolson viscosity's solves over tiles (ppe_compact.cu: rows for
the fluid, the other neighbours on the right-hand side) against the 8-byte
layout: a handful of fluid particles, odd sizes with one tile a block, several
tiles a block; both arithmetics.  One step from the same state, within the
bounds test_gpu_cn.py holds either layout to against the FP64 oracle."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_tiles import SCENES, _flow, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,niu,arith", [
    ("few rows", 1.0, "fast"), ("one tile a block", 1e-2, "exact"), ("one tile a block", 1.0, "fast"),
    ("several tiles a block", 1e-2, "fast")])
def test_cn_tiles_match_8_byte_layout(capi, name, niu, arith):
    pos, vel, nb2, nb1 = _flow(*SCENES[name], 0.01)
    p = _params(capi, 0.01, 5e-4)
    p.niu = niu
    out = []
    for layout in (0, -1):
        with capi.Simulation.from_arrays(p, pos, nb2, nb1, vel, method=capi.METHOD_SEMI_IMPLICIT, visc_implicit=1,
                                         arith=capi.ARITH_FAST if arith == "fast" else capi.ARITH_EXACT,
                                         ppe_layout=layout) as s:
            st = s.step(1)
            assert st.status == 0 and st.cg_relres <= 1e-8
            out.append(s.state(capi.ORDER_BY_ID))
    a, b = out
    assert np.abs(a["pos"] - b["pos"]).max() / np.abs(b["pos"]).max() < 1e-6
    assert rel_err(a["vel"], b["vel"]) < 1e-3
