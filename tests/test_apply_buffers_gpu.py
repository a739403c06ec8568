"""gbc_apply into every state of its result buffer (fresh pages, pages all there, some there, only read; in
place) on both sides of the 32 MB from which fresh pages are made resident beside the copies: the operator's
sites are those of a small call, the others keep the caller's values."""
import ctypes as C
import mmap

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [5, 6])  # 31.5 and 37.7 MB
def test_result_buffer_states(nrhs):
    dims = (8, 8, 16, 16)
    V = int(np.prod(dims))
    odd = S.parity(dims) == 1
    dp = lambda a: a.view(np.float64).ctypes.data_as(C.POINTER(C.c_double))
    x = np.stack([S.gaussian(dims, k, cb=1).reshape(V, 12) for k in range(nrhs)]).astype(np.complex128)
    ctx = G.Context(dims, 1 / (2 * 0.115) - 4, 1.0, t_boundary=-1, max_rhs=nrhs)
    try:
        ctx.load_gauge(G.gauge_synthetic(dims, 0.3, 5, t_boundary=-1))
        # FP64 of one right-hand side: its bits do not depend on how many there are
        want = np.concatenate([ctx.apply(G.OP_MEO, x[k:k + 1], 1, 1, G.PREC_DOUBLE)[:, odd] for k in range(nrhs)])

        def fresh():
            return np.frombuffer(mmap.mmap(-1, x.nbytes), np.complex128).reshape(x.shape)

        present, some, read = fresh(), fresh(), fresh()
        present[:] = 0.5 - 1j
        some[nrhs // 2] = 2.0
        assert not read.any()
        for name, out in (("fresh", fresh()), ("present", present), ("some", some), ("read", read), ("in place", x)):
            keep = out[:, ~odd].copy()
            assert ctx.lib.gbc_apply(ctx.h, G.OP_MEO, 1, 1, G.PREC_DOUBLE, nrhs, dp(out), dp(x)) == G.OK
            assert np.allclose(out[:, odd], want, rtol=0, atol=1e-13 * np.abs(want).max()), name
            assert np.array_equal(out[:, ~odd], keep), name
    finally:
        ctx.close()
