"""The free surface's two-level triangle scan at the edges of its blocks of
1,024 cubes: the triangles of the GPU's own vertex values, in the same number,
order of cubes and places as oracle/mc_oracle.py lists them."""
import numpy as np
import pytest

import mc_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 2), (34, 32, 2), (33, 33, 2), (42, 26, 2), (65, 9, 5), (65, 17, 9)])
def test_scan_blocks(capi, tmp_path, shape):
    from mps_solvers_b200 import scene
    sc = scene.small_tank(seed=5, interior=(20, 8, 16), fluid=(8, 8, 12), l0=0.02, dt=1e-4)
    d = str(tmp_path / "c")
    scene.write_case(d, sc)
    # vertices from inside the water to past its corner, so that cubes are cut
    s = 2 * sc.wall_layers
    origin = tuple((s + 0.25) * sc.l0 for _ in range(3))
    spacing = tuple(14.0 * sc.l0 / (n - 1) for n in shape)
    with capi.Simulation(d, method=capi.METHOD_EXPLICIT) as sim:
        sim.surface_setup(shape, origin, spacing, 100000)
        n = sim.surface_extract()
        pos, _ = sim.surface_triangles()
        values, iso = sim.surface_vertex_values()
    table = [list(t) for t in mo.build_table()]
    ref = mo.triangles(values.astype(np.float64), iso, origin, spacing, table)
    assert n == len(ref) and n > 0
    # points are float32 interpolations of coordinates below 0.5 m: a few
    # rounding steps of 3e-8, times the cancellation in n1 (iso - n2): 1e-5 m
    assert np.abs(pos - ref).max() < 1e-5
