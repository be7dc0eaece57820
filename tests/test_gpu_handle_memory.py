"""A batch and the Crank-Nicolson viscosity hold their matrices in one layout:
with the tiles they take no more device memory than with the 8-byte layout
(a tile's entries are 6 bytes for 8, plus its column list; 5 % covers the
lists of small scenes).  And the autotuner on a batch times the layout it has."""
import numpy as np
import pytest

from helpers import load_golden, write_golden_case
from test_gpu_tiles import _flow, _params

pytestmark = pytest.mark.gpu


def _used(make):
    import torch
    with make():  # what the driver keeps from a first use is not counted
        pass
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with make() as s:
        torch.cuda.synchronize()
        assert s.step(1).status == 0
        return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("learned", [False, True])
def test_batch_memory(capi, tmp_path, learned):
    import os
    from mps_solvers_b200 import scene
    dirs = []
    for k in range(3):
        dirs.append(str(tmp_path / str(k)))
        os.makedirs(dirs[-1])
        pos, vel, nb2, nb1 = _flow((41, 23, 29), (30, 20, 23), 0.01)
        prm = scene.Params(dim=3, dp=0.01, r0=2.1, rlap=4.0, cs=20.0, dt_max=5e-4, tt=1.0, max_dis=0.01)
        scene.write_input_dat(os.path.join(dirs[-1], "input.dat"), prm)
        scene.write_geo_dat(os.path.join(dirs[-1], "GEO.dat"), pos, nb2, nb1, vel)
    opt = dict(method=capi.METHOD_SEMI_IMPLICIT, arith=capi.ARITH_FAST,
               precond=capi.PRECOND_LEARNED if learned else capi.PRECOND_DIAGONAL)
    tiles, entries = (_used(lambda: capi.Simulation.batch(dirs, ppe_layout=lay, **opt)) for lay in (0, -1))
    assert tiles <= 1.05 * entries, (tiles, entries)


def test_viscosity_memory(capi):
    pos, vel, nb2, nb1 = _flow((41, 23, 29), (30, 20, 23), 0.01)
    used = {}
    for lay in (0, -1):
        for cn in (0, 1):
            used[lay, cn] = _used(lambda: capi.Simulation.from_arrays(
                _params(capi, 0.01, 5e-4), pos, nb2, nb1, vel, method=capi.METHOD_SEMI_IMPLICIT,
                arith=capi.ARITH_FAST, ppe_layout=lay, visc_implicit=cn))
    assert used[0, 1] - used[0, 0] <= 1.05 * (used[-1, 1] - used[-1, 0]), used


def test_autotune_a_batch(capi, tmp_path):
    dirs = [write_golden_case(load_golden("semi_tank"), str(tmp_path / f"s{k}")) for k in range(2)]
    for layout in (0, -1):
        with capi.Simulation.batch(dirs, method=capi.METHOD_SEMI_IMPLICIT, ppe_layout=layout) as s:
            rep = s.autotune(1)
            assert rep["ppe_compact"] == 0
            assert (rep["ppe_compact_ms"][0] > 0) == (layout == 0)
            assert (np.array(rep["ppe_ms"]) > 0).any() == (layout == -1)
            s.apply_tuning(rep)
            assert s.step(1).status == 0
            assert (s.scalars()["ppe_escaped"] >= 0) == (layout == 0)
