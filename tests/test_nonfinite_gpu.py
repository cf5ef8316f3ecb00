"""Cells, cotangents and coefficients at the edges of the number range, on
layouts that TMA refuses and with per-face tables: the same NaN and infinities
as the one-thread-per-face and one-thread-per-column kernels give, and the
same finite values."""
import numpy as np
import pytest

from gpu_util import to_dev
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
