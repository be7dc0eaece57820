"""Changing the PPE layout between a step and what reads the step's system.

mps_apply_tuning and mps_autotune change the layout of the steps that follow;
the system of the last step stays the one it was assembled as.  Loss and
gradients of the learned preconditioner, the exported matrix and the count of
far entries are the same before and after a switch, in both directions.

The same kernels run on the same arrays, so the matrix is equal; a gradient
is a sum of a few hundred blocks' partial sums by float atomics in any order,
which moves its entries by some 1e-6 of the largest (2^-24 a partial sum).
"""
import numpy as np
import pytest

from helpers import load_golden, write_golden_case

pytestmark = pytest.mark.gpu

TUNE = {"stage_threads": 256, "ppe_threads": 1024, "ppe_stored_weights": 1, "ppe_pipelined": 0}


def _sim(capi, tmp_path, layout):
    from mps_solvers_b200 import precond_weights
    d = write_golden_case(load_golden("semi_tank"), str(tmp_path / "s"))
    s = capi.Simulation(d, method=capi.METHOD_SEMI_IMPLICIT, precond=capi.PRECOND_LEARNED, ppe_layout=layout)
    s.set_precond_params(precond_weights.load())
    s.step(2)
    return s


def _switch(s, layout):
    s.apply_tuning({**TUNE, "ppe_compact": 1 if layout == -1 else 0})


@pytest.mark.parametrize("layout", [0, -1])
def test_training_after_a_layout_switch(capi, tmp_path, layout):
    with _sim(capi, tmp_path, layout) as s:
        loss, grad = s.precond_loss_grad(seed=7)
        _switch(s, layout)
        loss2, grad2 = s.precond_loss_grad(seed=7)
        assert abs(loss2 - loss) <= 1e-6 * abs(loss)
        assert np.abs(grad2 - grad).max() <= 1e-5 * np.abs(grad).max()
        assert s.step(1).cg_relres <= 1e-8


@pytest.mark.parametrize("layout", [0, -1])
def test_stencil_after_a_layout_switch(capi, tmp_path, layout):
    with _sim(capi, tmp_path, layout) as s:
        a, far = s.ppe_stencil(), s.scalars()["ppe_escaped"]
        _switch(s, layout)
        b = s.ppe_stencil()
        for f in ("row_start", "cols", "weights"):
            assert np.array_equal(a[f], b[f]), f
        assert s.scalars()["ppe_escaped"] == far
        s.step(1)
        assert (s.scalars()["ppe_escaped"] == -1) == (layout == 0)


def test_stencil_after_tuning_a_batch(capi, tmp_path):
    """The tuner's last timed step of a batch may be in the 8-byte layout."""
    dirs = [write_golden_case(load_golden("semi_tank"), str(tmp_path / f"s{k}")) for k in range(2)]
    with capi.Simulation.batch(dirs, method=capi.METHOD_SEMI_IMPLICIT) as s:
        s.autotune(1)
        st = s.ppe_stencil()
        assert st["cols"].max() < s.counts()["np"] and (st["weights"] > 0).all()
        n = len(st["row_start"]) - 1
        i = np.repeat(np.arange(n, dtype=np.int64), np.diff(st["row_start"].astype(np.int64)))
        j = st["cols"].astype(np.int64)
        assert np.array_equal(np.sort(i * n + j), np.sort(j * n + i))  # a symmetric pair set
        assert s.step(1).status == 0
