"""The warps' walk over the linked cells (mps_device.cuh: flat_batches) and the
tile layout's assembly on it (ppe_compact.cu), against sums over all pairs in
double precision: grids whose edges no power of two divides, cells with none,
one and a dozen particles, few rows and many.

A weight re/r - 1 comes from 2-ulp reciprocal square roots of r^2 (relative
error 1.5e-7 from the rounded differences): at most 5e-7 re/r.  A sum of up
to 20 weights a lane and 5 levels over the lanes adds 25 * 6e-8 of itself."""
import numpy as np
import pytest

from test_gpu_tiles import _flow, _params

pytestmark = pytest.mark.gpu


def _sums(pos, typ, re, skip_dummy):
    """sum of re/r and of the weights over the neighbours of every particle"""
    p = pos.astype(np.float64)
    near, w = np.zeros(len(p)), np.zeros(len(p))
    for a in range(0, len(p), 256):
        r = np.sqrt(((p[a:a + 256, None, :] - p[None]) ** 2).sum(-1))
        hit = (r < re) & (r > 0)
        if skip_dummy:
            hit &= (typ != 2)[None]
        k = np.where(hit, re / np.where(hit, r, 1.0), 0.0)
        near[a:a + 256] = k.sum(1)
        w[a:a + 256] = np.where(hit, k - 1.0, 0.0).sum(1)
    return near, w


@pytest.mark.parametrize("interior,fluid,layout", [
    ((9, 7, 9), (3, 3, 4), 0), ((9, 7, 9), (3, 3, 4), -1), ((23, 9, 17), (11, 7, 13), 0), ((17, 5, 31), (1, 1, 1), 0)])
def test_walk_sums(capi, interior, fluid, layout):
    pos, vel, nb2, nb1 = _flow(interior, fluid, 0.01)
    with capi.Simulation.from_arrays(_params(capi, 0.01, 5e-4), pos, nb2, nb1, vel, arith=capi.ARITH_FAST,
                                     method=capi.METHOD_SEMI_IMPLICIT, ppe_layout=layout) as s:
        assert s.step(1).status == 0
        t = s.ppe_snapshot()
    x, typ = t["pos4"][:, :3], t["pos4"][:, 3].view(np.uint32)
    near, w = _sums(x, typ, np.float64(np.float32(2.1 * 0.01)), False)
    some = typ != 2
    assert (np.abs(t["n"] - w) <= 2e-6 * near + 1e-6)[some].all()
    # the diagonal is the sum of the weights and one constant for all rows
    rows = t["is_row"] != 0
    near, w = _sums(x, typ, np.float64(np.float32(4.0 * 0.01)), True)
    c = -t["diag"][rows] - w[rows]
    assert rows.any() and (np.abs(c - np.median(c)) <= 4e-6 * near[rows].max() + 1e-6).all()
