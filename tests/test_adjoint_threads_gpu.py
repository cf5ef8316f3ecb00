"""The adjoint from several host threads at once: sweeps of different lengths
and with and without accumulation share kernels, whose shared-memory size
differs from call to call."""
import ctypes
import sys
import threading

import numpy as np
import pytest

from gpu_util import to_dev
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["arrays", "uniform"])
def test_lengths_and_accumulation(entry):
    """Every call succeeds, and the last one of each thread gives what it
    gives alone."""
    import torch
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import _lib, api, fields
    jobs, keep = [], []
    for m, acc in ((3, False), (199, False), (3, True), (199, True)) * 2:
        g = wsb.Grid(m, 1, 1, 1, 6)
        rng = np.random.default_rng(m)
        v = to_dev(rng.standard_normal(g.rs_shape(0)))
        gL, gR = (to_dev(rng.standard_normal(g.face_shape(0))) for _ in range(2))
        arrays = tuple(to_dev(x) for x in varying_coefficients(5, g.nc(0), seed=m))
        c = api.face_coefs(fields.uniform_weno_coefficients(5, 1)) if entry == "uniform" else api.coefs_struct(arrays)
        out = [torch.zeros(int(np.prod(g.rs_shape(0))), dtype=torch.float64, device="cuda") for _ in range(2)]
        stream = torch.cuda.Stream()
        gc = g.c()
        keep.append((v, gL, gR, arrays, c, gc))
        args = [(ctypes.byref(gc), 0, 5, wsb.F_MP | (wsb.F_ACCUMULATE if acc else 0), v.data_ptr(),
                 None if entry == "uniform" else ctypes.byref(c), ctypes.byref(c) if entry == "uniform" else None,
                 gL.data_ptr(), gR.data_ptr(), o.data_ptr(), int(stream.cuda_stream)) for o in out]
        assert wsb.lib().weno_sb_vjp_dev(*args[0]) == 0
        jobs.append((args[1], stream, out))
    torch.cuda.synchronize()
    errors = []

    def work(args, stream, out):
        for r in range(4000):
            rc = wsb.lib().weno_sb_vjp_dev(*args)
            if rc:
                errors.append((r, rc, _lib.last_error()))
                break
            if r % 200 == 0:
                stream.synchronize()
        stream.synchronize()
        with torch.cuda.stream(stream):
            out[1].zero_()
        wsb.lib().weno_sb_vjp_dev(*args)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    assert not errors, errors
    for _, _, out in jobs:
        assert torch.equal(out[0], out[1])
