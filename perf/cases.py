"""The workloads by which this library's speed is followed.

Each case is one time step's share of the WENO path as a program calls it:
x / y / z reconstruction sweeps on one block through the device-pointer
calls of `wenostandalone_b200.api`, the reference harness's drop-in sequence
(reshape, order-1 copy, reconstruction, limiter as separate calls), the
adjoint of the sweeps, or a batch of uneven blocks in one graph launch.
Fields, grids and coefficients are those of the harness driver, the
benchmark and the tests: smooth-plus-jump fields with noise, sinusoids with
a shock, uniform-grid, stretched-grid and harness coefficients.

`exact` restates the reference's formulas (wilfonba/WenoStandalone
inputs/weno_standalone.f90:281-1615) in plain torch FP64; for the adjoint it
differentiates them with torch.autograd.
"""
import functools
import math

import numpy as np
import torch

import wenostandalone_b200 as wsb
from wenostandalone_b200 import api, fields

BUFF = 6
SCHEMES = {"js": wsb.JS, "teno": wsb.TENO}
EPS, TENO_CT = 1e-16, 1e-5
HARNESS_OFFSETS = (0.03, 0.05, 0.07)


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _sweep(name, cells, v, order=5, scheme="js", coefs="uniform"):
    return dict(name=name, kind="sweep", nx=cells[0], ny=cells[1], nz=cells[2], v=v, order=order, scheme=scheme,
                coefs=coefs)


def listed():
    return [
        # a small block of an adaptive or strongly decomposed run: launches and host calls count
        _sweep("sweep5_16cubed", (16, 16, 16), 5),
        # the harness in x only at 64^3, mode weno5, scope full: reshape, order-1 copy, WENO5 from the
        # coefficient arrays, no limiter
        dict(name="dropin_weno5_x_64cubed", kind="dropin", nx=64, ny=64, nz=64, v=8, mode="weno5", dirs="x"),
        # the main workload: FP64 WENO5-JS + MP on one 200^3 block, reading the cell field directly
        _sweep("sweep5_200cubed", (200, 200, 200), 8),
        # the harness's full sequence at its default size (every kernel family, separate calls)
        dict(name="dropin_all_200cubed", kind="dropin", nx=200, ny=200, nz=200, v=8, mode="all", dirs="xyz"),
        # seventh order, for turbulence-resolving runs
        _sweep("sweep7_128cubed", (128, 128, 128), 5, order=7),
        # TENO weights on a block with odd extents (any decomposition of an odd grid gives some)
        _sweep("teno5_119x87x103", (119, 87, 103), 8, scheme="teno"),
        # WENO5-JS on a block with odd extents
        _sweep("sweep5_151x97x75", (151, 97, 75), 5),
        # a stretched grid: coefficients differ from face to face; mixed odd and even extents
        _sweep("stretched5_160x121x90", (160, 121, 90), 6, coefs="stretched"),
        # FP32 storage at 256^3 with 10 variables: reshape to FP32, then the sweep
        dict(name="mixed5_256cubed", kind="mixed", nx=256, ny=256, nz=256, v=10, order=5),
        # gradient of the three sweeps (design optimisation, data assimilation), uniform grid
        dict(name="vjp5_128cubed", kind="vjp", nx=128, ny=128, nz=128, v=5, order=5, scheme="js", coefs="uniform"),
        # the same on a stretched grid with odd extents
        dict(name="vjp5_stretched_97x80x65", kind="vjp", nx=97, ny=80, nz=65, v=5, order=5, scheme="js",
             coefs="stretched"),
        # uneven blocks of mixed order, x / y / z each, one graph launch
        dict(name="batch_24", kind="batch", blocks=24, lo=16, hi=112, shapes=96),
    ]


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "dropin", "mixed", "vjp", "vjp", "batch"])
    hi = {"sweep": 200, "dropin": 180, "mixed": 256, "vjp": 128, "batch": 112}[kind]
    if kind == "batch":
        return dict(kind="batch", blocks=rng.randint(4, 24), lo=16, hi=rng.randint(48, hi), shapes=rng.randrange(10**6))
    c = dict(kind=kind, nx=_extent(rng, 16, hi), ny=_extent(rng, 16, hi), nz=_extent(rng, 16, hi),
             v=rng.choice([1, 3, 5, 6, 8]))
    if kind == "dropin":
        return dict(c, mode=rng.choice(["weno5", "all"]), dirs="xyz")
    if kind == "mixed":
        return dict(c, order=rng.choice([3, 5, 7]))
    order = rng.choice([3, 5, 5, 5, 7])
    return dict(c, order=order, scheme=rng.choice(["js", "js", "teno"]) if order == 5 else "js",
                coefs=rng.choice(["uniform", "stretched"]))


# ---------------------------------------------------------------------------
# Inputs, and what a program keeps between calls
# ---------------------------------------------------------------------------
def _grid(c):
    return wsb.Grid(c["nx"] - 1, c["ny"] - 1, c["nz"] - 1, c["v"], BUFF, scheme=SCHEMES[c.get("scheme", "js")],
                    weno_eps=EPS, teno_CT=TENO_CT)


@functools.lru_cache(maxsize=None)
def _uniform(order):
    return fields.uniform_weno_coefficients(order, 1)


def _coefficients(kind, order, grid, d):
    """One direction's coefficient arrays on the host, in the reference's layouts."""
    if kind == "uniform":
        return _uniform(order)
    if kind == "harness":
        return fields.harness_coefficients(grid.nc(d), HARNESS_OFFSETS[d])
    cells = (grid.m_cells, grid.n_cells, grid.p_cells)[d] + 1
    return api.weno_coefficients(order, api.stretched_boundaries(cells, BUFF, centre=0.4 + 0.1 * d))


def _flat(a, device="cuda"):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).ravel(order="F"))).to(device)


def _on_device(host):
    return tuple(_flat(a) for a in host)


def _field(c, seed):
    args = (c["nx"] - 1, c["ny"] - 1, c["nz"] - 1, c["v"], BUFF)
    if c["kind"] == "mixed":
        return fields.sinusoid_shock_field_dev(*args, seed=seed)
    if c["kind"] == "vjp":
        return fields.sinusoid_shock_field_dev(*args, seed=seed, shock=False)
    return fields.smooth_jump_field_dev(*args, seed=seed)


def _size(shape):
    return int(np.prod(shape))


def _faces(grid, d, dtype=torch.float64):
    return torch.zeros(_size(grid.face_shape(d)), dtype=dtype, device="cuda")


def _cotangents(grid, d, seed):
    gen = torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) + d)
    n = _size(grid.face_shape(d))
    return [torch.randn(n, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2)]


def _blocks(c):
    """Block shapes of a batch: cells per axis uniform in lo..hi, order 3 / 5 / 7, JS or TENO weights."""
    rng = np.random.default_rng(c["shapes"])
    out = []
    for _ in range(c["blocks"]):
        cells = [int(x) for x in rng.integers(c["lo"], c["hi"] + 1, 3)]
        v, order = int(rng.choice([5, 8, 10])), int(rng.choice([3, 5, 7]))
        scheme = "js" if order != 5 else str(rng.choice(["js", "teno"]))
        out.append(dict(kind="sweep", nx=cells[0], ny=cells[1], nz=cells[2], v=v, order=order, scheme=scheme,
                        coefs="uniform"))
    return out


def prepare(case, seed):
    s = dict(kind=case["kind"], case=case)
    if case["kind"] == "batch":
        entries, outs = [], []
        for i, b in enumerate(_blocks(case)):
            g, v = _grid(b), _field(b, 100 * seed + i)
            # one allocation per block holds its six face-state arrays, each from a 256-byte boundary
            sizes = [(_size(g.face_shape(d)) + 31) // 32 * 32 for d in range(3)]
            pool = torch.zeros(2 * sum(sizes), dtype=torch.float64, device="cuda")
            outs.append(pool)
            at = 0
            for d in range(3):
                n = _size(g.face_shape(d))
                L, R = pool[at:at + n], pool[at + sizes[d]:at + sizes[d] + n]
                at += 2 * sizes[d]
                host = tuple(np.repeat(a, g.nc(d), axis=1 if a.shape == (5, 1) else 0) for a in _uniform(b["order"]))
                entries.append(dict(grid=g, dir=d, order=b["order"], flags=wsb.F_MP | wsb.F_FOLDED, v_in=v,
                                    coefs=_on_device(host), vL=L, vR=R))
        s.update(batch=api.Batch(entries), outs=outs)
        return s
    g = _grid(case)
    v = _field(case, seed)
    s.update(grid=g, v=v, order=case.get("order", 5))
    if case["kind"] == "mixed":
        s["rs"] = [torch.zeros(_size(g.rs_shape(d)), dtype=torch.float32, device="cuda") for d in range(3)]
        s["face"] = api.face_coefs(_uniform(case["order"]))
        s["out"] = [(_faces(g, d, torch.float32), _faces(g, d, torch.float32)) for d in range(3)]
        return s
    if case["kind"] == "vjp":
        s["cot"] = [_cotangents(g, d, seed) for d in range(3)]
        s["gv"] = torch.zeros_like(v)
    else:
        s["out"] = [(_faces(g, d), _faces(g, d)) for d in range(3)]
    if case["kind"] == "dropin":
        s["rs"] = [torch.zeros(_size(g.rs_shape(d)), dtype=torch.float64, device="cuda") for d in range(3)]
        s["dirs"] = ["xyz".index(x) for x in case["dirs"]]
        s["orders"] = [5] if case["mode"] == "weno5" else [3, 5, 7]
        s["mp"] = case["mode"] == "all"
        s["arrays"] = [_on_device(_coefficients("harness", 5, g, d)) for d in range(3)]
        s["coefs"] = [api.coefs_struct(a) for a in s["arrays"]]
    elif case["coefs"] == "uniform":
        s["face"] = api.face_coefs(_uniform(case["order"]))
    else:
        s["arrays"] = [_on_device(_coefficients("stretched", case["order"], g, d)) for d in range(3)]
        s["coefs"] = [api.coefs_struct(a) for a in s["arrays"]]
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].launch()
        return s["outs"]
    g, order = s["grid"], s["order"]
    if kind == "sweep":
        flags = wsb.F_MP | wsb.F_FOLDED
        for d in range(3):
            L, R = s["out"][d]
            if "face" in s:
                api.weno_uniform(g, d, order, s["v"], s["face"], L, R, flags=flags)
            else:
                api.weno(g, d, order, s["v"], s["coefs"][d], L, R, flags=flags)
        return s["out"]
    if kind == "mixed":
        for d in range(3):
            api.reshape(g, d, s["v"], s["rs"][d])
            api.weno_uniform(g, d, order, s["rs"][d], s["face"], *s["out"][d], flags=wsb.F_MP)
        return s["out"]
    if kind == "vjp":
        for d in range(3):
            flags = wsb.F_MP | wsb.F_FOLDED | (wsb.F_ACCUMULATE if d else 0)
            if "face" in s:
                api.vjp(g, d, order, s["v"], s["face"], *s["cot"][d], s["gv"], flags=flags, uniform=True)
            else:
                api.vjp(g, d, order, s["v"], s["coefs"][d], *s["cot"][d], s["gv"], flags=flags)
        return s["gv"]
    # the harness's order of calls: every reshape, every copy, then family by family
    for d in s["dirs"]:
        api.reshape(g, d, s["v"], s["rs"][d])
    for d in s["dirs"]:
        api.order1_copy(g, d, s["v"], *s["out"][d])
    for o in s["orders"]:
        for d in s["dirs"]:
            api.weno(g, d, o, s["rs"][d], s["coefs"][d], *s["out"][d])
    if s["mp"]:
        for d in s["dirs"]:
            api.preserve_monotonicity(g, d, s["rs"][d], *s["out"][d])
    return {"rs": [s["rs"][d] for d in s["dirs"]], "states": [s["out"][d] for d in s["dirs"]]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
_FLOPS = {3: 45, 5: 110, 7: 210}  # per face: differences, indicators, weights, both states
_MP_FLOPS = 45


def _one_work(g, d, order, size, mp=True):
    """(bytes, operations) of one sweep: the stencil window of every column read once, both states written."""
    ns, c1, c2 = g.extents(d)
    nf, half = (ns, 1) if order == 3 else (ns - 6, 2 if order == 5 else 3)
    if mp:
        half = max(half, 2)
    cols = c1 * c2 * g.v_size
    return (nf + 2 * half + 2 * nf) * cols * size, nf * cols * (_FLOPS[order] + (_MP_FLOPS if mp else 0))


def work(case):
    if case["kind"] == "batch":
        parts = [work(b) for b in _blocks(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    g = _grid(case)
    total, ops = 0, 0
    for d in range(3) if case["kind"] != "dropin" else ["xyz".index(x) for x in case["dirs"]]:
        rs, faces = _size(g.rs_shape(d)) * 8, _size(g.face_shape(d)) * 8
        if case["kind"] == "dropin":
            # separate calls: reshape, copy into both states, each family, the limiter in place
            total += 2 * rs + 3 * faces
            for o in ([5] if case["mode"] == "weno5" else [3, 5, 7]):
                b, f = _one_work(g, d, o, 8, mp=False)
                total, ops = total + b, ops + f
            if case["mode"] == "all":
                total, ops = total + rs + 4 * faces, ops + _MP_FLOPS * faces // 8
        else:
            b, f = _one_work(g, d, case["order"], 4 if case["kind"] == "mixed" else 8)
            if case["kind"] == "mixed":
                # the reshape reads the FP64 field and writes the FP32 one
                b += rs + rs // 2
            if case["kind"] == "vjp":
                # the field and two cotangents are read, the gradient is added to (written first)
                b += rs * (2 if d else 1)
                f *= 3
            total, ops = total + b, ops + f
    return {"bytes": total, "flops": ops}


# ---------------------------------------------------------------------------
# The reference's formulas in FP64 torch
# ---------------------------------------------------------------------------
def _column_view(v, d):
    """v (z, y, x) of one variable -> (c2, c1, sweep cells) of direction d (f90:281-330)."""
    if d == 0:
        return v[3:-3, 3:-3, :]
    if d == 1:
        return v[3:-3, :, 3:-3].permute(0, 2, 1)
    return v[:, 3:-3, 3:-3].permute(2, 1, 0)


def _per_face(host, nfaces, first):
    """Coefficient arrays expanded to one set per face first .. first + nfaces - 1 (core index clamped)."""
    pL, pR, dL, dR, bc = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in host)
    c = (torch.arange(nfaces, device="cuda") + first - 3).clamp(0, pL.shape[0] - 1)
    return pL[c], pR[c], dL[:, c], dR[:, c], bc[c]


def _weno(x, order, scheme, host):
    """(vL, vR, first face) of the faces a sweep writes; x (..., ns + 6)."""
    R = (order + 1) // 2
    S = R - 1
    ns = x.shape[-1] - 6
    first, nf = (0, ns) if order == 3 else (3, ns - 6)
    pL, pR, dL, dR, bc = _per_face(host, nf, first)
    at = lambda k: x[..., first + 3 + k:first + 3 + k + nf]  # noqa: E731
    v0 = at(0)
    D = {k: at(k + 1) - at(k) for k in range(-S, S)}
    beta, offL, offR = [], [], []
    for r in range(R):
        t = [D[S - 1 - r - s] for s in range(S)]
        b, i = 0.0, 0
        for a in range(S):
            for e in range(a, S):
                b = b + bc[:, r, i] * t[a] * t[e]
                i += 1
        beta.append(b + EPS)
        offL.append(sum(pL[:, r, s] * t[s] for s in range(S)))
        offR.append(sum(pR[:, r, s] * t[s] for s in range(S)))
    if scheme == "teno":
        tau = (beta[2] - beta[0]).abs()
        a = [(1.0 + tau / b) ** 6 for b in beta]
        total = a[0] + a[1] + a[2]
        w = [torch.where(y / total < TENO_CT, 0.0, 1.0) for y in a]
    else:
        w = [1.0 / (b * b) for b in beta]
    out = []
    for ideal, off in ((dL, offL), (dR, offR)):
        # WENO7 pairs weight q with coefficient row 3 - q (f90:1462-1488)
        al = [ideal[3 - r if order == 7 else r] * w[r] for r in range(R)]
        total = sum(al)
        out.append(v0 + sum(al[r] * off[r] for r in range(R)) / total)
    return out[0], out[1], first


def _minmod(a, b):
    m, M = torch.minimum(a.abs(), b.abs()), torch.maximum(a.abs(), b.abs())
    t = 4.0 * m - M
    return torch.where((a * b > 0) & (t > 0), torch.sign(a) * torch.minimum(t, m), torch.zeros_like(a))


def _limit(x, L, R):
    """The monotonicity limiter on the core faces (f90:1544-1615); L, R on faces 3 .. ns - 4."""
    nf = x.shape[-1] - 12
    at = lambda k: x[..., 6 + k:6 + k + nf]  # noqa: E731
    m2, m1, v0, p1, p2 = (at(k) for k in range(-2, 3))
    dm, dc, dp = v0 + m2 - 2.0 * m1, p1 + m1 - 2.0 * v0, p2 + v0 - 2.0 * p1
    mA, mB = _minmod(dm, dc), _minmod(dc, dp)

    def side(s, near, far, md, lc):
        UL = v0 - 2.0 * (far - v0)
        MD = 0.5 * (v0 + near - md)
        LC = v0 - 0.5 * (far - v0) + 4.0 / 3.0 * lc
        lo = torch.maximum(torch.minimum(torch.minimum(v0, near), MD), torch.minimum(torch.minimum(v0, UL), LC))
        hi = torch.minimum(torch.maximum(torch.maximum(v0, near), MD), torch.maximum(torch.maximum(v0, UL), LC))
        return torch.minimum(torch.maximum(s, lo), hi)

    return side(L, m1, p1, mA, mB), side(R, p1, m1, mB, mA)


def _write(out, x, order, scheme, host, mp):
    """The faces one sweep writes into out = (vL, vR) (..., ns)."""
    L, R, first = _weno(x, order, scheme, host)
    if mp:
        core = slice(3 - first, 3 - first + x.shape[-1] - 12)
        l, r = _limit(x, L[..., core], R[..., core])
        L[..., core], R[..., core] = l, r
    n = L.shape[-1]
    out[0][..., first:first + n], out[1][..., first:first + n] = L, R


def _exact_states(c, v, d, grid, host, mp=True):
    ns, c1, c2 = grid.extents(d)
    out = [torch.zeros((grid.v_size, c2, c1, ns), dtype=torch.float64, device="cuda") for _ in range(2)]
    for q in range(grid.v_size):
        _write((out[0][q], out[1][q]), _column_view(v[q], d), c["order"], c.get("scheme", "js"), host, mp)
    return out[0].reshape(-1), out[1].reshape(-1)


def exact(case, seed):
    if case["kind"] == "batch":
        outs = []
        for i, b in enumerate(_blocks(case)):
            states = [x for pair in exact(b, 100 * seed + i) for x in pair]
            pad = [(x.numel() + 31) // 32 * 32 for x in states]
            pool = torch.zeros(sum(pad), dtype=torch.float64, device="cuda")
            at = 0
            for x, n in zip(states, pad):
                pool[at:at + x.numel()] = x
                at += n
            outs.append(pool)
        return outs
    g = _grid(case)
    flat = _field(case, seed)
    if case["kind"] == "mixed":
        flat = flat.float().double()
    N = g.N
    v = flat.reshape(case["v"], N[2] + 6, N[1] + 6, N[0] + 6)
    if case["kind"] in ("sweep", "mixed"):
        return [_exact_states(case, v, d, g, _coefficients(case.get("coefs", "uniform"), case["order"], g, d))
                for d in range(3)]
    if case["kind"] == "vjp":
        cot = [_cotangents(g, d, seed) for d in range(3)]
        hosts = [_coefficients(case["coefs"], case["order"], g, d) for d in range(3)]
        out = torch.zeros_like(v)
        for d in range(3):
            ns, c1, c2 = g.extents(d)
            gL, gR = (x.reshape(g.v_size, c2, c1, ns) for x in cot[d])
            for q in range(g.v_size):
                x = v[q].clone().requires_grad_(True)
                col = _column_view(x, d)
                L, R, first = _weno(col, case["order"], case["scheme"], hosts[d])
                n = L.shape[-1]
                k = 3 - first
                l, r = _limit(col, L[..., k:k + ns - 6], R[..., k:k + ns - 6])
                L, R = (torch.cat([y[..., :k], z, y[..., k + ns - 6:]], -1) for y, z in ((L, l), (R, r)))
                f = (L * gL[q][..., first:first + n]).sum() + (R * gR[q][..., first:first + n]).sum()
                out[q] += torch.autograd.grad(f, x)[0]
        return out.reshape(-1)
    rs, states = [], []
    for d in ["xyz".index(x) for x in case["dirs"]]:
        ns, c1, c2 = g.extents(d)
        host = _coefficients("harness", 5, g, d)
        full = torch.stack([_column_view(v[q], d) for q in range(g.v_size)])
        rs.append(full.reshape(-1))
        out = [full[..., 3:-3].clone(), full[..., 3:-3].clone()]
        for q in range(g.v_size):
            for o in [5] if case["mode"] == "weno5" else [3, 5, 7]:
                _write((out[0][q], out[1][q]), full[q], o, "js", host, False)
            if case["mode"] == "all":
                core = slice(3, ns - 3)
                l, r = _limit(full[q], out[0][q][..., core], out[1][q][..., core])
                out[0][q][..., core], out[1][q][..., core] = l, r
        states.append((out[0].reshape(-1), out[1].reshape(-1)))
    return {"rs": rs, "states": states}
