"""Layouts that TMA refuses keep the precision of the one-thread-per-face
kernels: FP32 storage of the families those computed in FP64 (WENO3-JS and
the TENO weights) rounds once, and TENO cutoffs fall on the side on which the
divisions put them."""
import numpy as np
import pytest

from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu

# Nd = cells + 2 buff + 1 = 33, 35, 31: no direction's rows are multiples of
# 4 floats or of 2 doubles
M, N, P, BUFF = 20, 22, 18, 6


@pytest.mark.parametrize("order,scheme", [(3, 0), (5, 3), (7, 3)])
def test_fp32_storage_rounds_once(oracle_mod, order, scheme):
    """Without the limiter a state is the FP64 state rounded to FP32: within
    half an ulp, 2^-24 of its size, of the oracle, plus the FP64 bar."""
    import torch
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    # (the reference's WENO7-TENO has alpha(4) = (1 + tau / eps)^6, which cuts
    # every stencil at the usual eps)
    eps = 0.05 if order == 7 else 1e-16
    g = wsb.Grid(M, N, P, 2, BUFF, scheme=scheme, weno_eps=eps)
    rng = np.random.default_rng(6)
    vf = rng.standard_normal((M + 19, N + 19, P + 19, 2)).astype(np.float32).astype(np.float64)
    vf = np.asfortranarray(vf)
    for d in range(3):
        coefs = fields.uniform_weno_coefficients(order, g.nc(d))
        rs = oracle_mod.reshape(vf, M, N, P, BUFF, d)
        ref = oracle_mod.order1_copy(vf, M, N, P, BUFF, d)
        got = [to_dev(x, torch.float32) for x in ref]
        oracle_mod.reconstruct(rs, coefs, order, scheme=scheme, eps=eps, vL=ref[0], vR=ref[1])
        api.weno_uniform(g, d, order, to_dev(rs, torch.float32), coefs, *got)
        sure = np.ones(ref[0].shape, dtype=bool)
        if scheme == 3:
            sure = oracle_mod.teno_margin(rs, coefs, order, eps=eps) > 1e-10
            assert sure.mean() > 0.99
        for x, r in zip(got, ref):
            e = np.abs(from_dev(x, g.face_shape(d)) - r)
            assert np.all((e <= 2.0 ** -24 * np.abs(r) + 1e-12 * np.abs(r).max())[sure]), (d, e[sure].max())


def _omega(x, order, coefs, eps):
    """Normalised TENO alphas (f90:578-606, 1491-1506) of the core faces of
    one column set x (ns + 6, ...), with uniform coefficients."""
    R = (order + 1) // 2
    beta_coef = np.asarray(coefs[4])[0]
    nf = x.shape[0] - 12
    at = lambda k: x[6 + k:6 + k + nf]  # noqa: E731
    S = R - 1
    D = {k: at(k + 1) - at(k) for k in range(-S, S)}
    b = []
    for r in range(R):
        t, v, i = [D[S - 1 - r - s] for s in range(S)], eps, 0
        for p in range(S):
            for q in range(p, S):
                v = v + beta_coef[r, i] * t[p] * t[q]
                i += 1
        b.append(v)
    if order == 7:
        b = b[::-1] + [np.full_like(b[0], eps)]
        tau = np.abs(b[4] - b[3])
    else:
        tau = np.abs(b[2] - b[0])
    a = np.stack([(1.0 + tau / y) ** 6 for y in b])
    return (a / a.sum(0))[:R]


@pytest.mark.parametrize("order", [5, 7])
@pytest.mark.parametrize("entry", ["uniform", "arrays"])
def test_teno_cutoffs(monkeypatch, order, entry):
    """Cutoffs placed 2^-46 and 2^-45.5 beside the weight of one stencil of
    one face: near enough for ratios from one Newton step (2^-46, six of them
    in the power) to land on the wrong side, far enough for ratios within a
    few ulp.  States and (WENO5) gradients equal those of the divisions."""
    import wenostandalone_b200 as wsb
    from wenostandalone_b200 import api, fields
    eps = 0.05 if order == 7 else 1e-16
    vf = fields.smooth_jump_field(M, N, P, 2, BUFF, seed=9)
    g0 = wsb.Grid(M, N, P, 2, BUFF)
    coefs = fields.uniform_weno_coefficients(order, g0.nc(0))
    x = vf[:, 3:-3, 3:-3, :]
    w = _omega(x, order, coefs, eps)
    rng = np.random.default_rng(2)
    ok = np.flatnonzero((w > 1e-4) & (w < 0.2))
    targets = w.ravel()[rng.choice(ok, 12, replace=False)]
    v = to_dev(vf)
    shape = g0.face_shape(0)
    gL, gR = (to_dev(rng.standard_normal(shape)) for _ in range(2))
    c = coefs if entry == "uniform" else tuple(to_dev(a) for a in coefs)
    for t in targets:
        for delta in (-2.0 ** -45.5, -2.0 ** -46, 2.0 ** -46, 2.0 ** -45.5):
            g = wsb.Grid(M, N, P, 2, BUFF, scheme=3, weno_eps=eps, teno_CT=float(t * (1.0 + delta)))
            out = []
            for kernel in ("auto", "generic"):
                monkeypatch.setenv("WENO_SB_KERNEL", kernel)
                L, R, gv = to_dev(np.zeros(shape)), to_dev(np.zeros(shape)), to_dev(np.zeros(vf.shape))
                run = api.weno_uniform if entry == "uniform" else api.weno
                run(g, 0, order, v, c, L, R, flags=wsb.F_FOLDED)
                if order == 5:
                    api.vjp(g, 0, order, v, c, gL, gR, gv, flags=wsb.F_FOLDED, uniform=entry == "uniform")
                out.append((L, R, gv))
            for got, ref, tol in zip(*out, (1e-12, 1e-12, 1e-9)):
                assert float((got - ref).abs().max()) <= tol * float(ref.abs().max()), (t, delta, tol)
