"""The pool of the per-face tables gives its memory back: many large tables,
made and freed, leave no more in use than the pool may keep."""
import numpy as np
import pytest

from gpu_util import to_dev
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu


def test_tables_are_freed():
    """1.8 MB a table (4013 faces of 448 bytes), 200 calls: 360 MB if none
    were freed, against the 64 MB the pool may keep."""
    import torch
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(4000, 1, 1, 1, 6)
    assert g.face_shape(0)[0] == 4013
    v = to_dev(fields.smooth_jump_field(4000, 1, 1, 1, 6, seed=2))
    c = tuple(to_dev(x) for x in varying_coefficients(7, g.nc(0), seed=1))
    L, R = (torch.zeros(int(np.prod(g.face_shape(0))), dtype=torch.float64, device="cuda") for _ in range(2))
    free = []
    for n in (1, 200):
        for _ in range(n):
            api.weno(g, 0, 7, v, c, L, R, flags=wsb.F_FOLDED)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] >= free[0] - (64 << 20), free
