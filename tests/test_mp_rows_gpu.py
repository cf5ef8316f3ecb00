"""The standalone limiter at the smallest sweeps (1 to 3 core faces: a warp's
faces span many columns) and at remainders of its 64-face steps, bit for bit
against the general kernel's fused limiter (the same arithmetic per face)."""
import numpy as np
import pytest

from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(0, 0, 0, 1, 3), (2, 1, 0, 2, 3), (60, 7, 5, 3, 6), (51, 12, 20, 1, 6)])
def test_small_sweeps(monkeypatch, dims, dtype):
    import torch
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    monkeypatch.setenv("WENO_SB_KERNEL", "generic")
    m, n, p, nv, buff = dims
    tdt = torch.float64 if dtype == "fp64" else torch.float32
    g = wsb.Grid(m, n, p, nv, buff)
    # rough data, so that the limiter acts on many faces
    v = to_dev(fields.smooth_jump_field(m, n, p, nv, buff, seed=6, noise=0.3))
    coefs = fields.uniform_weno_coefficients(5, 1)
    for d in range(3):
        rs = torch.empty(int(np.prod(g.rs_shape(d))), dtype=tdt, device="cuda")
        api.reshape(g, d, v, rs)
        out = []
        for flags in (wsb.F_MP, 0):
            L, R = (torch.full((int(np.prod(g.face_shape(d))),), 7.0, dtype=tdt, device="cuda") for _ in range(2))
            api.weno_uniform(g, d, 5, rs, coefs, L, R, flags=flags)
            out.append((L, R))
        raw = [x.clone() for x in out[1]]
        api.preserve_monotonicity(g, d, rs, *out[1])
        for want, got, before in zip(*out, raw):
            assert torch.equal(want, got), d
            assert not torch.equal(got, before), d
