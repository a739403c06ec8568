"""gbc_apply_meo_noalloc under the caller's stream capture, where its second launch may be placed early: replays
of the graph on new inputs give bit for bit what direct calls give, for grids on both sides of the size
up to which that is done (304 blocks), with the output apart from the input and on it."""
import ctypes as C

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.1


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("dims", [(4, 4, 4, 6), (8, 8, 8, 8), (8, 8, 10, 12)])  # 24, 256 and 480 blocks
def test_graph_replays_equal_direct_calls(dims, in_place):
    import torch
    V = int(np.prod(dims))
    u = G.gauge_synthetic(dims, 0.3, 11, t_boundary=-1)
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=1)
    try:
        ctx.load_gauge(u)
        clov, inv, _, _ = ctx.get_clover()
    finally:
        ctx.close()
    links, tc, ti = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (u, clov, inv))
    fn = G.load().gbc_apply_meo_noalloc
    fn.argtypes = [C.POINTER(G.Geom), C.POINTER(G.Action)] + [C.c_void_p] * 3 + [C.c_int] + [C.c_void_p] * 3
    geom, act = G.Geom((C.c_int * 4)(*dims), -1), G.Action(MASS, CSW, CSW, 0, 1.0, 1.0, 3, 0, 0.0)

    def call(x, y, stream):  # y = M~ x
        assert fn(C.byref(geom), C.byref(act), links.data_ptr(), tc.data_ptr(), ti.data_ptr(), 1, y.data_ptr(),
                  x.data_ptr(), stream.cuda_stream) == 0

    xs = [torch.from_numpy(np.ascontiguousarray(S.gaussian(dims, 4 + k).reshape(V, 12))).cuda() for k in range(3)]
    want = []
    for x in xs:
        y = x.clone()
        call(x, y, torch.cuda.current_stream())
        want.append(y)
    torch.cuda.synchronize()
    src = torch.zeros_like(xs[0])
    dst = src if in_place else torch.zeros_like(src)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):  # back to back: the second call's first launch follows the early-placed one
            call(src, dst, torch.cuda.current_stream())
    odd = torch.from_numpy(S.parity(dims) == 1).cuda()
    for x, y in zip(xs, want):
        src.copy_(x)
        graph.replay()
        torch.cuda.synchronize()
        if in_place:  # applied twice
            z = y.clone()
            call(y, z, torch.cuda.current_stream())
            torch.cuda.synchronize()
            y = z
        assert torch.equal(dst[odd], y[odd]) and bool(dst[odd].abs().sum() > 0)
