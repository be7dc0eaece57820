"""The cell sorts with an output over their input: a caller that needs the
positions no more may let the permutation or the cells take their place.
The same tables as with arrays of their own, for one to three radix passes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["mps_cell_sort_dev", "mps_cell_sort_dev_noalloc"])
@pytest.mark.parametrize("cells", [(5, 4, 3), (20, 10, 15), (80, 40, 25)])
@pytest.mark.parametrize("over", ["perm", "cell"])
def test_output_over_the_positions(capi, fn, cells, over):
    import torch
    n = 70001
    g = capi.mps_grid(left=0.0, back=0.0, bottom=0.0, cell_size=0.1, cdx=cells[0], cdy=cells[1], cdz=cells[2],
                      ncells=cells[0] * cells[1] * cells[2], dim=3)
    rng = np.random.default_rng(1)
    pos = np.zeros((n, 4), np.float32)
    for a in range(3):
        pos[:, a] = rng.uniform(-0.05, 0.1 * cells[a] + 0.05, n)
    res = []
    for shared in (False, True):
        x = torch.from_numpy(pos).cuda()
        out = {k: torch.empty(m, dtype=torch.int32, device="cuda")
               for k, m in (("perm", n), ("cell", n), ("start", g.ncells), ("end", g.ncells), ("nin", 1))}
        if shared:
            out[over] = x.view(torch.int32).flatten()[n // 2:n // 2 + n]
        st = getattr(capi.lib(), fn)(C.c_void_p(x.data_ptr()), n, C.byref(g), *[C.c_void_p(out[k].data_ptr()) for k in
                                     ("perm", "cell", "start", "end", "nin")], None)
        assert st == 0
        torch.cuda.synchronize()
        res.append({k: v.cpu().numpy() for k, v in out.items()})
    for k in res[0]:
        assert np.array_equal(res[0][k], res[1][k]), k
