"""Cells, cotangents and coefficients at the edges of the number range, on
layouts that TMA refuses and with per-face tables: the same NaN and infinities
as the one-thread-per-face and one-thread-per-column kernels give, and the
same finite values."""
import numpy as np
import pytest

from gpu_util import from_dev, rel_err, to_dev
from test_adjoint_gpu import TOL_AD
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu

M, N, P, BUFF = 20, 22, 18, 6  # Nd 33, 35, 31


def _put(a, value, seed, count=40):
    rng = np.random.default_rng(seed)
    a[tuple(rng.integers(0, s, count) for s in a.shape)] = value


def _same(got, ref, tol):
    got, ref = got.cpu().numpy(), ref.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], ref[inf])
    fin = np.isfinite(ref)
    err = np.abs(got[fin] - ref[fin])
    # (huge cells: relative to the value; others: to the field's size)
    assert np.all(err <= tol * np.maximum(np.abs(ref[fin]), 10.0)), float(err.max())


def _coefs(wsb, entry, order, g, d):
    from wenostandalone_b200 import fields
    host = (fields.uniform_weno_coefficients(order, g.nc(d)) if entry == "uniform"
            else varying_coefficients(order, g.nc(d), seed=d))
    return [np.array(c) for c in host]


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e200])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("order,scheme", [(3, 0), (5, 0), (5, 1), (5, 2), (5, 3), (7, 0), (7, 3)])
def test_sweeps(monkeypatch, order, scheme, entry, bad):
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(M, N, P, 2, BUFF, scheme=scheme)
    vf = fields.smooth_jump_field(M, N, P, 2, BUFF, seed=5)
    _put(vf, bad, 3)
    v = to_dev(vf)
    for d in range(3):
        c = _coefs(wsb, entry, order, g, d)
        out = []
        for kernel in ("auto", "generic"):
            monkeypatch.setenv("WENO_SB_KERNEL", kernel)
            L, R = to_dev(np.zeros(g.face_shape(d))), to_dev(np.zeros(g.face_shape(d)))
            if entry == "uniform":
                api.weno_uniform(g, d, order, v, tuple(c), L, R, flags=wsb.F_FOLDED | wsb.F_MP)
            else:
                api.weno(g, d, order, v, tuple(to_dev(a) for a in c), L, R, flags=wsb.F_FOLDED | wsb.F_MP)
            out.append((L, R))
        for got, ref in zip(*out):
            _same(got, ref, 1e-12)


def _gradients(monkeypatch, wsb, g, d, entry, vf, c, gL, gR, g0, mp=True):
    from wenostandalone_b200 import api
    out = []
    flags = wsb.F_FOLDED | wsb.F_ACCUMULATE | (wsb.F_MP if mp else 0)
    for kernel in ("auto", "generic"):
        monkeypatch.setenv("WENO_SB_KERNEL", kernel)
        gv = to_dev(g0)
        cs = tuple(c) if entry == "uniform" else tuple(to_dev(a) for a in c)
        api.vjp(g, d, 5, to_dev(vf), cs, to_dev(gL), to_dev(gR), gv, flags=flags, uniform=entry == "uniform")
        out.append(gv)
    return out


@pytest.mark.parametrize("where,bad", [("cell", np.nan), ("cell", np.inf), ("cell", 1e200), ("cotangent", np.nan),
                                       ("cotangent", np.inf), ("gradient", np.nan), ("gradient", np.inf)])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("scheme", [0, 3])
def test_adjoint(monkeypatch, scheme, entry, where, bad):
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import fields
    g = wsb.Grid(M, N, P, 2, BUFF, scheme=scheme)
    for d in range(3):
        for mp in (False, True):
            rng = np.random.default_rng(12)
            vf = fields.smooth_jump_field(M, N, P, 2, BUFF, seed=5)
            gL, gR = rng.standard_normal(g.face_shape(d)), rng.standard_normal(g.face_shape(d))
            g0 = rng.standard_normal(vf.shape)
            for a in {"cell": [vf], "cotangent": [gL, gR], "gradient": [g0]}[where]:
                _put(a, bad, 4, 25)
            c = _coefs(wsb, entry, 5, g, d)
            got, ref = _gradients(monkeypatch, wsb, g, d, entry, vf, c, gL, gR, g0, mp)
            # gradients of rough cells reach some hundreds: TOL_AD of that
            _same(got, ref, 100 * TOL_AD)


@pytest.mark.parametrize("cells", [(20, 22, 18), (21, 23, 19)])  # odd rows; rows that suit TMA
@pytest.mark.parametrize("scale", [2.0 ** -600, 2.0 ** -300, 2.0 ** 300])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("scheme", [0, 3])
def test_scaled_ideal_weights(scheme, entry, scale, cells):
    """The weights are normalised, so a common factor of the ideal weights
    changes nothing."""
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    m, n, p = cells
    g = wsb.Grid(m, n, p, 1, BUFF, scheme=scheme)
    vf = fields.sinusoid_shock_field(m, n, p, 1, BUFF, seed=4, shock=False)
    rng = np.random.default_rng(5)
    for d in range(3):
        gL, gR = (to_dev(rng.standard_normal(g.face_shape(d))) for _ in range(2))
        out = []
        for f in (1.0, scale):
            c = _coefs(wsb, entry, 5, g, d)
            c[2] *= f
            c[3] *= f
            cs = tuple(c) if entry == "uniform" else tuple(to_dev(a) for a in c)
            gv = to_dev(np.zeros(vf.shape))
            api.vjp(g, d, 5, to_dev(vf), cs, gL, gR, gv, flags=wsb.F_FOLDED | wsb.F_MP, uniform=entry == "uniform")
            out.append(from_dev(gv, vf.shape))
        assert rel_err(out[1], out[0]) <= TOL_AD, d


@pytest.mark.parametrize("entry", ["uniform", "arrays"])
@pytest.mark.parametrize("zero", [0, 1, 2])
def test_teno_zero_ideal_weight(monkeypatch, entry, zero):
    """A face whose kept stencils have no weight on one side has NaN there
    only, as with the divisions."""
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import fields
    g = wsb.Grid(M, N, P, 2, BUFF, scheme=3)
    vf = fields.smooth_jump_field(M, N, P, 2, BUFF, seed=5)
    rng = np.random.default_rng(12)
    for d in range(3):
        gL, gR = rng.standard_normal(g.face_shape(d)), rng.standard_normal(g.face_shape(d))
        c = _coefs(wsb, entry, 5, g, d)
        c[2][zero] = 0.0
        c[3][2 - zero] = 0.0
        got, ref = _gradients(monkeypatch, wsb, g, d, entry, vf, c, gL, gR, np.zeros(vf.shape))
        _same(got, ref, 100 * TOL_AD)
