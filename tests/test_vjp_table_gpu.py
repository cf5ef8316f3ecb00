"""The marching adjoint with per-face coefficient arrays (WENO5): one chunk,
remainders of the chunk, of the segment and of the 32-column tile, the
longest sweep whose table fits into shared memory and the first that does not
(another kernel), faces marked by a negative ideal weight; accumulated, in
both layouts, against the dual-number oracle."""
import numpy as np
import pytest

from gpu_util import from_dev, rel_err, to_dev
from test_adjoint_gpu import TOL_AD
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu

# cells per axis minus one, variables; a sweep has 12 faces more than cells and
# the table holds sweeps of up to 214 faces
DIMS = [(1, 2, 9, 1), (33, 30, 8, 2), (201, 4, 5, 1), (4, 201, 3, 1), (3, 2, 201, 1), (202, 2, 3, 1)]


def _slow_wave(shape):
    """Resolved on every grid: the weights stay near the ideal ones, so a
    small negative weight cancels nothing."""
    i, j, k, q = np.indices(shape)
    return np.asfortranarray(2.0 + np.sin(0.05 * (i + 2 * j + 3 * k) + q))


@pytest.mark.parametrize("scheme", [0, 3])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("negative", [False, True])
def test_per_face_adjoint(oracle_mod, dims, scheme, negative):
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    m, n, p, nv = dims
    g = wsb.Grid(m, n, p, nv, 6, scheme=scheme)
    vf = fields.sinusoid_shock_field(m, n, p, nv, 6, seed=4, shock=False)
    if negative:
        vf = _slow_wave(vf.shape)
    rng = np.random.default_rng(29)
    for d in range(3):
        coefs = varying_coefficients(5, g.nc(d), seed=d)
        if negative:
            for ideal in coefs[2:4]:
                ideal[0, ::7] = -1e-6
        rs = oracle_mod.reshape(vf, m, n, p, 6, d)
        gL = np.asfortranarray(rng.standard_normal(g.face_shape(d)))
        gR = np.asfortranarray(rng.standard_normal(g.face_shape(d)))
        ref = oracle_mod.vjp(rs, coefs, 5, gL, gR, scheme=scheme, mp=True)
        dev = tuple(to_dev(c) for c in coefs)
        g0 = np.asfortranarray(rng.standard_normal(rs.shape))
        gv = to_dev(g0)
        api.vjp(g, d, 5, to_dev(rs), dev, to_dev(gL), to_dev(gR), gv, flags=wsb.F_MP | wsb.F_ACCUMULATE)
        assert rel_err(from_dev(gv, rs.shape), g0 + ref) <= TOL_AD, (d, "accumulated")
        # the field's own layout: the sweep's cells are those of the reshaped
        # field, all others receive nothing
        folded = to_dev(np.full(vf.shape, np.nan, order="F"))
        api.vjp(g, d, 5, to_dev(vf), dev, to_dev(gL), to_dev(gR), folded, flags=wsb.F_MP | wsb.F_FOLDED)
        got = from_dev(folded, vf.shape)
        assert rel_err(oracle_mod.reshape(got, m, n, p, 6, d), ref) <= TOL_AD, (d, "folded")
        assert np.count_nonzero(got) <= ref.size
