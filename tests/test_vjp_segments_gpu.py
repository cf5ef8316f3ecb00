"""The adjoint of small blocks: columns cut into segments of cells (a segment
starts early, so that every face that reaches its cells is counted once), at
the smallest sweep and at remainders of the segment and of the column tile;
accumulated onto a gradient, against the dual-number oracle."""
import numpy as np
import pytest

from gpu_util import from_dev, rel_err, to_dev
from test_adjoint_gpu import TOL_AD, TOL_AD3
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [3, 5, 7])
@pytest.mark.parametrize("entry", ["arrays", "uniform"])
@pytest.mark.parametrize("dims", [(0, 1, 2, 1, 3), (2, 3, 4, 1, 3), (38, 33, 50, 1, 6)])
def test_small_blocks(oracle_mod, dims, entry, order):
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    m, n, p, nv, buff = dims
    g = wsb.Grid(m, n, p, nv, buff)
    vf = fields.smooth_jump_field(m, n, p, nv, buff, seed=8)
    rng = np.random.default_rng(17)
    for d in range(3):
        coefs = (fields.uniform_weno_coefficients(order, g.nc(d)) if entry == "uniform"
                 else varying_coefficients(order, g.nc(d), seed=d))
        rs = oracle_mod.reshape(vf, m, n, p, buff, d)
        gL = np.asfortranarray(rng.standard_normal(g.face_shape(d)))
        gR = np.asfortranarray(rng.standard_normal(g.face_shape(d)))
        g0 = np.asfortranarray(rng.standard_normal(rs.shape))
        ref = g0 + oracle_mod.vjp(rs, coefs, order, gL, gR, mp=True)
        gv = to_dev(g0)
        fl = wsb.F_MP | wsb.F_ACCUMULATE
        if entry == "uniform":
            api.vjp(g, d, order, to_dev(rs), coefs, to_dev(gL), to_dev(gR), gv, flags=fl, uniform=True)
        else:
            api.vjp(g, d, order, to_dev(rs), tuple(to_dev(c) for c in coefs), to_dev(gL), to_dev(gR), gv, flags=fl)
        assert rel_err(from_dev(gv, rs.shape), ref) <= (TOL_AD3 if order == 3 else TOL_AD), d
