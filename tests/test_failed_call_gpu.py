"""A call that fails leaves the caller's result buffer as it was and the next call works: a network application
whose wait for the tensor cores gave up (a buffer larger than the 2 MB below which no helper thread
runs), and a smearing whose allocation the device refuses."""
import ctypes as C

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu


def _dp(a):
    return a.view(np.float64).ctypes.data_as(C.POINTER(C.c_double))


def test_failed_network_leaves_the_result_alone(monkeypatch):
    dims = (8, 8, 8, 16)
    ctx = G.Context(dims, 1 / (2 * 0.115) - 4, 1.0, t_boundary=-1, max_rhs=2)
    try:
        ctx.load_gauge(G.gauge_synthetic(dims, 0.3, 5, t_boundary=-1))
        monkeypatch.setenv("GBC_TC_QUIT_WARP", "0")
        ctx.precond_init(hidden=12, layers=2, seed=1)
        monkeypatch.delenv("GBC_TC_QUIT_WARP")
        x = np.stack([S.gaussian(dims, 8 + k, cb=1).reshape(-1, 12) for k in range(2)]).astype(np.complex128)
        out = np.full(x.shape, (1 + 2j) / 3)
        assert ctx.lib.gbc_precond_apply(ctx.h, 2, _dp(out), _dp(x)) != 0
        assert np.all(out == (1 + 2j) / 3)
        ctx.precond_init(hidden=12, layers=2, seed=1)
        assert ctx.lib.gbc_precond_apply(ctx.h, 2, _dp(out), _dp(x)) == 0
        assert np.array_equal(out, ctx.precond_apply(x))
    finally:
        ctx.close()


def test_refused_smearing_does_not_fail_the_next_call():
    """A lattice of 2.5 TB of links: the allocation is refused before any host buffer is touched."""
    dims = (4, 4, 4, 8)
    ctx = G.Context(dims, 1 / (2 * 0.115) - 4, 1.0, t_boundary=-1, max_rhs=1)
    try:
        ctx.load_gauge(G.gauge_synthetic(dims, 0.3, 5, t_boundary=-1))
        x = S.gaussian(dims, 8, cb=1).reshape(1, -1, 12).astype(np.complex128)
        want = ctx.apply(G.OP_MEO, x)
        u = np.full((64, 4, 3, 3), (1 + 2j) / 3)
        out = np.full((64, 4, 3, 3), (1 + 2j) / 3)
        geom = G.Geom((C.c_int * 4)(256, 256, 256, 256), 1)
        assert ctx.lib.gbc_stout_smear(C.byref(geom), 1, 0.1, (C.c_int * 4)(1, 1, 1, 1), _dp(u), _dp(out)) == G.ERR_CUDA
        assert np.all(out == (1 + 2j) / 3)
        assert np.array_equal(ctx.apply(G.OP_MEO, x), want)
    finally:
        ctx.close()
