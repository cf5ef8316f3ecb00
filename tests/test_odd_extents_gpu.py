"""Sweeps whose face rows or field rows are not 16-byte multiples: odd
extents, extents not a multiple of 4 in FP32, and arrays that start at an odd
element.  The marching engines take them with per-lane loads and plain
stores; every family against the CPU oracle, at the smallest sweep they
cover (9 odd faces) and with tile remainders of 1, 3 and 5 columns."""
import numpy as np
import pytest

from gpu_util import from_dev, rel_err, to_dev
from test_parity_gpu import _check, varying_coefficients

pytestmark = pytest.mark.gpu

# (m, n, p, v, buff): Nd = cells + 2 buff + 1
DIMS = [(2, 2, 2, 1, 3), (20, 22, 18, 2, 6), (86, 19, 24, 1, 6)]
FAMILIES = [(3, 0), (5, 0), (5, 1), (5, 2), (5, 3), (7, 0), (7, 3)]


@pytest.fixture(scope="module")
def wsb():
    import torch
    assert torch.cuda.is_available()
    import wenostandalone_b200 as w
    w.lib()
    return w


def _shifted(flat, off):
    """The values of `flat` in a buffer that starts `off` elements late."""
    import torch
    buf = torch.full((flat.numel() + off,), float("nan"), dtype=flat.dtype, device=flat.device)
    buf[off:] = flat
    return buf[off:]


def _case(wsb, oracle_mod, dims, d, order, scheme, folded, entry, mp, dtype, off):
    import torch
    from wenostandalone_b200 import api, fields
    m, n, p, nv, buff = dims
    g = wsb.Grid(m, n, p, nv, buff, scheme=scheme)
    vf = fields.smooth_jump_field(m, n, p, nv, buff, seed=5)
    if dtype == torch.float32:
        vf = vf.astype(np.float32).astype(np.float64)
    coefs = (fields.uniform_weno_coefficients(order, g.nc(d)) if entry == "uniform"
             else varying_coefficients(order, g.nc(d), seed=d + order))
    rs = oracle_mod.reshape(np.asfortranarray(vf), m, n, p, buff, d)
    Lr, Rr = oracle_mod.order1_copy(np.asfortranarray(vf), m, n, p, buff, d)
    oracle_mod.reconstruct(rs, coefs, order, scheme=scheme, vL=Lr, vR=Rr)
    if mp:
        oracle_mod.preserve_monotonicity(rs, Lr, Rr)
    L, R = (_shifted(to_dev(x, dtype), off) for x in oracle_mod.order1_copy(np.asfortranarray(vf), m, n, p, buff, d))
    src = _shifted(to_dev(vf if folded else rs, dtype), off)
    flags = (wsb.F_FOLDED if folded else 0) | (wsb.F_MP if mp else 0)
    if entry == "uniform":
        api.weno_uniform(g, d, order, src, coefs, L, R, flags=flags)
    else:
        api.weno(g, d, order, src, tuple(to_dev(c) for c in coefs), L, R, flags=flags)
    margin = oracle_mod.teno_margin(rs, coefs, order) if scheme == 3 else None
    return from_dev(L, g.face_shape(d)), from_dev(R, g.face_shape(d)), Lr, Rr, margin


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("folded", [False, True])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("order,scheme", FAMILIES)
def test_fp64(wsb, oracle_mod, order, scheme, entry, folded, off):
    """off 1 on the middle block only (its extents are odd too): arrays from
    an odd element, so that the bases are 8-byte aligned."""
    import torch
    for dims in DIMS if off == 0 else DIMS[1:2]:
        for d in range(3):
            for mp in (False, True):
                Lg, Rg, Lr, Rr, mg = _case(wsb, oracle_mod, dims, d, order, scheme, folded, entry, mp, torch.float64,
                                           off)
                _check(Lg, Rg, Lr, Rr, scheme, (dims, d, mp), mg)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("order", [3, 5, 7])
def test_fp32_bulk(wsb, oracle_mod, order, off):
    """FP32-bulk with the limiter: 1e-6 against the oracle on the same
    FP32-rounded field (the bar of the even-extent tests)."""
    import torch
    for dims in DIMS[1:] + [(21, 23, 25, 1, 6)]:
        for d in range(3):
            Lg, Rg, Lr, Rr, _ = _case(wsb, oracle_mod, dims, d, order, 0, False, "uniform", True, torch.float32, off)
            assert rel_err(Lg, Lr) <= 1e-6 and rel_err(Rg, Rr) <= 1e-6, (dims, d)
