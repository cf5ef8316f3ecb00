"""Per-face calls captured into a CUDA graph: replays follow the inputs, and
calls that never put memory into the graph still put none."""
import numpy as np
import pytest

from gpu_util import to_dev
from test_parity_gpu import varying_coefficients

pytestmark = pytest.mark.gpu

M, N, P, BUFF = 21, 20, 18, 6


def _shifted(flat, off):
    import torch
    buf = torch.zeros(flat.numel() + off, dtype=flat.dtype, device=flat.device)
    buf[off:] = flat
    return buf[off:]


def _captured(call):
    """(replay, node types) of the graph of one call; NaN where a node type
    cannot be read."""
    import torch
    from cuda.bindings import runtime as rt
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    ok = rt.cudaError_t.cudaSuccess
    (e,) = rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
    assert e == ok
    try:
        call(int(s.cuda_stream))
    finally:
        e, graph = rt.cudaStreamEndCapture(s.cuda_stream)
    assert e == ok
    _, _, n = rt.cudaGraphGetNodes(graph)
    e, nodes, n = rt.cudaGraphGetNodes(graph, n)
    assert e == ok and n > 0
    types = [rt.cudaGraphNodeGetType(x)[1] for x in nodes]
    e, ex = rt.cudaGraphInstantiate(graph, 0)
    assert e == ok

    def replay():
        (err,) = rt.cudaGraphLaunch(ex, s.cuda_stream)
        assert err == ok
        s.synchronize()

    return replay, types


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("order,scheme", [(3, 0), (5, 0), (5, 3), (7, 0)])
def test_sweep(order, scheme, off):
    """Fields from an odd element (off 1) took kernels without a table, whose
    graphs hold no memory."""
    import torch
    import wenostandalone_b200 as wsb
    from cuda.bindings import runtime as rt
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(M, N, P, 2, BUFF, scheme=scheme)
    c = tuple(to_dev(x) for x in varying_coefficients(order, g.nc(0), seed=3))
    v = _shifted(to_dev(fields.smooth_jump_field(M, N, P, 2, BUFF, seed=1)), off)
    L, R, L1, R1 = (torch.zeros(int(np.prod(g.face_shape(0))), dtype=torch.float64, device="cuda") for _ in range(4))
    flags = wsb.F_FOLDED | wsb.F_MP
    api.weno(g, 0, order, v, c, L1, R1, flags=flags)
    torch.cuda.synchronize()
    replay, types = _captured(lambda s: api.weno(g, 0, order, v, c, L, R, flags=flags, stream=s))
    if off:
        assert rt.cudaGraphNodeType.cudaGraphNodeTypeMemAlloc not in types
    for seed in (1, 2):
        v.copy_(to_dev(fields.smooth_jump_field(M, N, P, 2, BUFF, seed=seed)))
        api.weno(g, 0, order, v, c, L1, R1, flags=flags)
        torch.cuda.synchronize()
        replay()
        for a, b in ((L, L1), (R, R1)):
            assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max()), seed


@pytest.mark.parametrize("scheme", [0, 3])
def test_adjoint(scheme):
    import torch
    import wenostandalone_b200 as wsb
    from cuda.bindings import runtime as rt
    from test_adjoint_gpu import TOL_AD
    from wenostandalone_b200 import api, fields
    g = wsb.Grid(M, N, P, 1, BUFF, scheme=scheme)
    c = tuple(to_dev(x) for x in varying_coefficients(5, g.nc(0), seed=3))
    rng = np.random.default_rng(4)
    gL, gR = (to_dev(rng.standard_normal(g.face_shape(0))) for _ in range(2))
    v = to_dev(fields.smooth_jump_field(M, N, P, 1, BUFF, seed=1))
    a, b = torch.zeros_like(v), torch.zeros_like(v)
    flags = wsb.F_FOLDED | wsb.F_MP
    api.vjp(g, 0, 5, v, c, gL, gR, b, flags=flags)
    torch.cuda.synchronize()
    replay, types = _captured(lambda s: api.vjp(g, 0, 5, v, c, gL, gR, a, flags=flags, stream=s))
    assert rt.cudaGraphNodeType.cudaGraphNodeTypeMemAlloc not in types
    for seed in (1, 2):
        v.copy_(to_dev(fields.smooth_jump_field(M, N, P, 1, BUFF, seed=seed)))
        api.vjp(g, 0, 5, v, c, gL, gR, b, flags=flags)
        torch.cuda.synchronize()
        replay()
        assert float((a - b).abs().max()) <= TOL_AD * float(b.abs().max()), seed
