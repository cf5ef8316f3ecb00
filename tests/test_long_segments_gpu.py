"""Odd layouts with enough columns that a warp's segment holds several chunks
of 8 faces: the sector-aligned stores between a segment's first and last
chunk, the tiles refilled behind them, whole columns of the adjoint; against
the CPU oracle on every element, outputs poisoned with NaN."""
import functools

import numpy as np
import pytest

from gpu_util import from_dev, nan_dev, rel_err, to_dev
from test_adjoint_gpu import TOL_AD, _scatter_to_vf
from test_parity_gpu import _check, varying_coefficients

pytestmark = pytest.mark.gpu

# Nd 151, 163, 45: 20 000 - 74 000 columns a sweep, segments of 5 to 11 chunks
# on 148 SMs
M, N, P, V, BUFF = 138, 150, 32, 3, 6


@functools.lru_cache(maxsize=None)
def _field():
    from wenostandalone_b200 import fields
    return fields.smooth_jump_field(M, N, P, V, BUFF, seed=11)


def _coefs(entry, order, nc, d):
    from wenostandalone_b200 import fields
    return (fields.uniform_weno_coefficients(order, nc) if entry == "uniform"
            else varying_coefficients(order, nc, seed=d + order))


def _late(flat, off):
    """The values of `flat` in a buffer that starts `off` elements late."""
    import torch
    buf = torch.empty(flat.numel() + off, dtype=flat.dtype, device=flat.device)
    buf[off:] = flat
    return buf[off:]


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("order,scheme", [(3, 0), (5, 0), (5, 1), (5, 2), (5, 3), (7, 0), (7, 3)])
def test_sweeps(oracle_mod, order, scheme, entry, d):
    """off: elements the field, vL and vR start late (vR alone: bases that
    differ by 8 bytes)."""
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api
    g = wsb.Grid(M, N, P, V, BUFF, scheme=scheme)
    vf = _field()
    coefs = _coefs(entry, order, g.nc(d), d)
    rs = oracle_mod.reshape(vf, M, N, P, BUFF, d)
    nan = np.full(g.face_shape(d), np.nan, order="F")
    Lr, Rr = oracle_mod.reconstruct(rs, coefs, order, scheme=scheme, vL=nan.copy(order="F"), vR=nan.copy(order="F"))
    margin = oracle_mod.teno_margin(rs, coefs, order) if scheme == 3 else None
    oracle_mod.preserve_monotonicity(rs, Lr, Rr)
    cs = coefs if entry == "uniform" else tuple(to_dev(c) for c in coefs)
    for folded, off in ((False, (0, 0, 0)), (True, (0, 0, 1)), (True, (1, 1, 1)), (False, (1, 0, 1))):
        src = _late(to_dev(vf if folded else rs), off[0])
        L, R = (_late(nan_dev(g.face_shape(d)), o) for o in off[1:])
        flags = wsb.F_MP | (wsb.F_FOLDED if folded else 0)
        (api.weno_uniform if entry == "uniform" else api.weno)(g, d, order, src, cs, L, R, flags=flags)
        _check(from_dev(L, g.face_shape(d)), from_dev(R, g.face_shape(d)), Lr, Rr, scheme, (d, folded, off), margin)


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("scheme", [0, 3])
def test_adjoint(oracle_mod, scheme, entry, d):
    """Resolved data: two correct gradients agree to TOL_AD there."""
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(M, N, P, V, BUFF, scheme=scheme)
    vf = fields.sinusoid_shock_field(M, N, P, V, BUFF, seed=4, shock=False)
    coefs = _coefs(entry, 5, g.nc(d), d)
    rs = oracle_mod.reshape(vf, M, N, P, BUFF, d)
    rng = np.random.default_rng(19)
    gL, gR = (np.asfortranarray(rng.standard_normal(g.face_shape(d))) for _ in range(2))
    ref = oracle_mod.vjp(rs, coefs, 5, gL, gR, scheme=scheme, mp=True)
    ref_vf = _scatter_to_vf(oracle_mod, vf.shape, M, N, P, BUFF, d, ref)
    cs = coefs if entry == "uniform" else tuple(to_dev(c) for c in coefs)
    for folded in (False, True):
        x, r = (vf, ref_vf) if folded else (rs, ref)
        g0 = np.asfortranarray(rng.standard_normal(r.shape))
        for acc in (False, True):
            gv = to_dev(g0) if acc else nan_dev(r.shape)
            flags = wsb.F_MP | (wsb.F_FOLDED if folded else 0) | (wsb.F_ACCUMULATE if acc else 0)
            api.vjp(g, d, 5, to_dev(x), cs, to_dev(gL), to_dev(gR), gv, flags=flags, uniform=entry == "uniform")
            got, want = from_dev(gv, r.shape), r + g0 if acc else r
            assert rel_err(got, want) <= TOL_AD, (folded, acc)
            # cells outside the sweep: exactly nothing added
            if folded:
                out = np.ones(r.shape, dtype=bool)
                s = [slice(3, -3)] * 3
                s[d] = slice(None)
                out[tuple(s)] = False
                assert np.array_equal(got[out], g0[out] if acc else np.zeros(int(out.sum())))
