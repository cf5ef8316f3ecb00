"""The per-face tables of concurrent calls: several host threads, each on its
own stream with its own coefficients, share the library's table pool."""
import threading

import numpy as np
import pytest

from gpu_util import to_dev
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [3, 5, 7])
def test_tables_of_concurrent_streams(order):
    """Results equal those of the same calls made one after the other, and
    the device's free memory does not shrink from round to round."""
    import torch
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(39, 30, 21, 2, 6)
    v = to_dev(fields.smooth_jump_field(39, 30, 21, 2, 6, seed=4))
    n_thr, n_rep = 4, 12

    def outputs():
        return [torch.zeros(int(np.prod(g.face_shape(0))), dtype=torch.float64, device="cuda") for _ in range(2)]

    coefs = [tuple(to_dev(c) for c in varying_coefficients(order, g.nc(0), seed=k)) for k in range(n_thr)]
    want = []
    for k in range(n_thr):
        L, R = outputs()
        api.weno(g, 0, order, v, coefs[k], L, R, flags=wsb.F_FOLDED | wsb.F_MP)
        torch.cuda.synchronize()
        want.append((L, R))
    got = [[outputs() for _ in range(n_rep)] for _ in range(n_thr)]
    torch.cuda.synchronize()
    free, errors = [], []

    def work(k):
        try:
            s = torch.cuda.Stream()
            for r in range(n_rep):
                api.weno(g, 0, order, v, coefs[k], *got[k][r], flags=wsb.F_FOLDED | wsb.F_MP,
                         stream=int(s.cuda_stream))
                if r % 3 == k % 3:
                    s.synchronize()
            s.synchronize()
        except Exception as e:  # reported by the main thread
            errors.append(e)

    for _ in range(2):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(n_thr)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert not errors, errors
    for k in range(n_thr):
        for L, R in got[k]:
            assert torch.equal(L, want[k][0]) and torch.equal(R, want[k][1])
    assert free[1] >= free[0] - (64 << 20), free  # what the pool may keep
