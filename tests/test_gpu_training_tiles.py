"""Training of the learned preconditioner on systems of a few to a few
hundred rows: partly filled 64-row tiles of the dense layers and partly filled
batches of 32 stencil entries.  Loss and gradients against the float64 oracle
at test_gpu_precond.py's tolerances."""
import numpy as np
import pytest

from test_gpu_precond import random_params, sim_and_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("interior,fluid", [((9, 6, 9), (3, 3, 4)), ((10, 7, 10), (5, 4, 5)), ((13, 7, 11), (7, 5, 7))])
def test_gradients_match_cpu_oracle(capi, tmp_path, interior, fluid):
    import precond_oracle as po
    from mps_solvers_b200 import scene
    d = str(tmp_path / "c")
    scene.write_case(d, scene.small_tank(seed=4, interior=interior, fluid=fluid, l0=0.02, dt=1e-4))
    w = random_params(capi, 2)
    s, system = sim_and_system(capi, d, w, steps=2)
    with s:
        loss, grad = s.precond_loss_grad(seed=5)
    ref = system.loss(w, 5)
    assert abs(loss - ref) <= 1e-5 + 1e-4 * abs(ref)
    rng = np.random.default_rng(3)
    for _ in range(2):
        v = rng.standard_normal(len(w))
        v /= np.linalg.norm(v)
        fd = po.directional_fd(system, w, v, 5, h=1e-3)
        an = float(grad.astype(np.float64) @ v)
        assert abs(fd - an) <= 2e-3 * max(abs(fd), 1e-6) + 1e-7
