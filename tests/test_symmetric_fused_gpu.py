"""The symmetric operator's fused second step (out = in - 1/4 A_oo^-1 D_oe t [+ twist]) at ragged block
edges, in every storage precision, and its fused reductions in BiCGStab solves.  Operators against the CPU
oracle with the tolerances of test_symmetric_gpu.py's precisions (1e-12, 1e-5, 5e-3); solutions by the
oracle's FP64 residual."""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.1


def _setup(dims):
    from oracle import Oracle, OracleOp
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 21), (1, 1, 1, -1))
    return u, OracleOp(dims, u, MASS, CSW)


@pytest.mark.parametrize("dims,nrhs", [((2, 2, 2, 6), 1), ((6, 6, 6, 10), 3), ((4, 6, 4, 6), 12)])
def test_operator(dims, nrhs):
    from oracle import oracle as O
    u, op = _setup(dims)
    V = int(np.prod(dims))
    odd = S.parity(dims) == 1
    xs = np.stack([S.gaussian(dims, 60 + k).reshape(V, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs)
    try:
        ctx.load_gauge(u)
        for prec, tol in ((G.PREC_DOUBLE, 1e-12), (G.PREC_SINGLE, 1e-5), (G.PREC_HALF, 5e-3)):
            for isign in (1, -1):
                got = ctx.apply(G.OP_SYM, xs, isign, 1, prec)
                for k in (0, nrhs - 1):
                    want = op.apply(O.OP_SYM, xs[k], isign)
                    assert np.linalg.norm((got[k] - want)[odd]) < tol * np.linalg.norm(want[odd]), (prec, isign, k)
    finally:
        ctx.close()


@pytest.mark.parametrize("prec", [G.PREC_HALF, G.PREC_SINGLE, G.PREC_DOUBLE], ids=["half", "single", "double"])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_bicgstab(nrhs, prec):
    from oracle import oracle as O
    dims = (6, 4, 6, 10)
    u, op = _setup(dims)
    chi = np.stack([S.z2_noise(dims, 7 + k, cb=1).reshape(-1, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs, sloppy_precision=prec)
    try:
        ctx.load_gauge(u)
        psi, _, rc = ctx.solve(chi, solver=G.SOLVER_BICGSTAB, system=G.SYS_SYM, rsd_target=1e-10, delta=0.01,
                               inner_tol=1e-5, sloppy_precision=prec)
    finally:
        ctx.close()
    assert rc == 0
    for k in range(nrhs):
        r = chi[k] - op.apply(O.OP_SYM, psi[k])
        assert np.sqrt(op.norm2(r) / op.norm2(chi[k])) <= 1.05e-10
