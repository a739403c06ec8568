"""Results handed back in host buffers: the sites a call does not own keep the caller's values whatever
state the buffer's pages are in, in-place calls work, and a context that loads one gauge field after
another (its packed fields are kept) gives what a fresh context gives.

Sizes on both sides of the 2 MB below which no helper thread runs.  Solutions against the oracle's FP64
residual; everything else is exact."""
import ctypes as C

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.0


def _context(dims, u, **kw):
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=4, **kw)
    ctx.load_gauge(u)
    return ctx


def _dp(a):
    return a.view(np.float64).ctypes.data_as(C.POINTER(C.c_double))


@pytest.mark.parametrize("dims,nrhs", [((4, 4, 4, 4), 1), ((8, 8, 8, 16), 2)])
def test_even_sites_survive(dims, nrhs):
    from oracle import Oracle, OracleOp
    from oracle import oracle as O
    u = Oracle().apply_bc(dims, Oracle().gauge_hot(dims, 0.3, 3), (1, 1, 1, -1))
    op = OracleOp(dims, u, MASS, CSW)
    V = int(np.prod(dims))
    odd = S.parity(dims) == 1
    chi = np.stack([S.z2_noise(dims, 2 + k, cb=1).reshape(V, 12) for k in range(nrhs)])
    ctx = _context(dims, u)
    try:
        for fresh in (True, False):
            psi = np.zeros(chi.shape, np.complex128)
            keep = np.zeros(chi.shape, np.complex128)
            if not fresh:
                keep = np.random.default_rng(1).standard_normal(chi.shape) + 0j
                psi[:] = keep
            p = G.SolveParams(G.SOLVER_MIXED, G.SYS_MEO, 1e-10, 10000, 0.1, 10.0, 0, 0.0, 0, 16, 0, 1, 0)
            res = (G.Result * nrhs)()
            assert ctx.lib.gbc_solve(ctx.h, C.byref(p), nrhs, _dp(psi), _dp(chi), res) == G.OK
            assert np.array_equal(psi[:, ~odd], keep[:, ~odd])
            for k in range(nrhs):
                x = psi[k] * odd[:, None]
                r = chi[k] - op.apply(O.OP_MEO, x)
                assert np.sqrt(op.norm2(r) / op.norm2(chi[k])) <= 1.05e-10
            # shifted systems: one buffer per shift
            ns = 3
            outs = [keep[0].copy() if not fresh else np.zeros((V, 12), np.complex128) for _ in range(ns)]
            pp = (C.POINTER(C.c_double) * ns)(*[_dp(o) for o in outs])
            sh = (C.c_double * ns)(0.01, 0.1, 1.0)
            rs = (G.Result * ns)()
            p = G.SolveParams(G.SOLVER_CG, G.SYS_MDAGM, 1e-10, 10000, 0.1, 10.0, G.PREC_SINGLE, 0.0, 0, 16, 0, 1, 0)
            assert ctx.lib.gbc_solve_multishift(ctx.h, C.byref(p), ns, sh, None, pp, _dp(chi[0]), rs) == G.OK
            for q in range(ns):
                assert np.array_equal(outs[q][~odd], keep[0][~odd])
                x = outs[q] * odd[:, None]
                y = op.apply(O.OP_MDAGM, x)
                r = (chi[0] - y - sh[q] * x) * odd[:, None]
                assert np.sqrt(op.norm2(r) / op.norm2(chi[0])) <= 1.05e-10
    finally:
        ctx.close()


@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (8, 8, 8, 16)])
def test_network_in_place(dims):
    u = G.gauge_synthetic(dims, 0.3, 5, t_boundary=-1)
    ctx = _context(dims, u)
    try:
        ctx.precond_init(hidden=12, layers=2, seed=1)
        x = S.gaussian(dims, 8, cb=1).reshape(1, -1, 12).astype(np.complex128).copy()
        want = ctx.precond_apply(x)
        assert ctx.lib.gbc_precond_apply(ctx.h, 1, _dp(x), _dp(x)) == G.OK
        assert np.array_equal(x, want)
    finally:
        ctx.close()


def test_reload_gauge_matches_fresh_context():
    dims = (4, 6, 4, 6)
    us = [G.gauge_synthetic(dims, 0.3, k, t_boundary=-1) for k in (1, 2)]
    us.insert(1, us[0] * 1.01)  # not SU(3): the 12-real planes fall back to 18 reals and come back
    x = S.gaussian(dims, 8).reshape(1, -1, 12)
    one = _context(dims, us[0])
    try:
        for u in us:
            one.load_gauge(u)
            fresh = _context(dims, u)
            try:
                assert np.allclose(one.logdet(), fresh.logdet(), rtol=1e-14, atol=0)
                for op in (G.OP_MEO, G.OP_SYM):
                    for prec in (G.PREC_DOUBLE, G.PREC_SINGLE, G.PREC_HALF):
                        a, b = one.apply(op, x, 1, 1, prec), fresh.apply(op, x, 1, 1, prec)
                        # the two contexts may have tuned different FP32 / fp16 launch shapes
                        tol = {G.PREC_DOUBLE: 0.0, G.PREC_SINGLE: 1e-5, G.PREC_HALF: 1e-2}[prec]
                        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b), (op, prec)
            finally:
                fresh.close()
    finally:
        one.close()


@pytest.mark.parametrize("nrhs", [1, 9, 10])
def test_reductions_on_both_sides_of_one_wave(nrhs):
    """128 blocks per right-hand side: 9 end inside the kernel, 10 in a launch of their own."""
    dims = (16, 16, 16, 16)
    u = G.gauge_synthetic(dims, 0.3, 1, t_boundary=-1)
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=10)
    try:
        ctx.load_gauge(u)
        odd = S.parity(dims) == 1
        f = np.stack([S.gaussian(dims, 20 + k, cb=1).reshape(-1, 12) for k in range(nrhs)]).astype(np.complex128)
        for _ in range(3):  # the counters are left at zero
            got = ctx.blas(G.BLAS_NORM2, [f])
            want = (np.abs(f[:, odd]) ** 2).sum((1, 2))
            assert np.allclose(got[:, 0], want, rtol=1e-12)
    finally:
        ctx.close()
