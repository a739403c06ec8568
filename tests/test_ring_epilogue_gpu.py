"""The fp16 ring kernel's epilogue operands, which come through its ring: solves whose stencil runs on one of
its launch shapes (GBC_SHAPE 9 to 11), with the |M psi|^2 of CGNE and the (r0, v), (t, s), (t, t) of BiCGStab
summed in the epilogue, at ragged last blocks and lattices of less than a block.  Solutions by the oracle's
FP64 residual."""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.0


@pytest.mark.parametrize("solver", [G.SOLVER_MIXED, G.SOLVER_BICGSTAB], ids=["cgne", "bicgstab"])
@pytest.mark.parametrize("dims,nrhs,mu", [((2, 4, 2, 6), 1, None), ((6, 6, 6, 10), 3, 0.05)], ids=["48", "1080x3-twisted"])
@pytest.mark.parametrize("shape", [9, 10, 11])
def test_solves(shape, dims, nrhs, mu, solver, monkeypatch):
    from oracle import Oracle, OracleOp
    from oracle import oracle as O
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 78), (1, 1, 1, -1))
    op = OracleOp(dims, u, MASS, CSW, twisted_m=mu)
    chi = np.stack([S.z2_noise(dims, 40 + k, cb=1).reshape(-1, 12) for k in range(nrhs)])
    monkeypatch.setenv("GBC_SHAPE", str(shape))
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs, twisted_m=mu)
    try:
        ctx.load_gauge(u)
        psi, res, rc = ctx.solve(chi, solver=solver, rsd_target=1e-10, delta=0.01 if solver == G.SOLVER_BICGSTAB else 0.1)
        ran = [line for line in ctx.tune_report().splitlines() if line.startswith("prec=2 ")]
    finally:
        ctx.close()
    assert rc == 0
    assert ran and all("pair=2 (GBC_SHAPE)" in line for line in ran), ran
    for k in range(nrhs):
        r = chi[k] - op.apply(O.OP_MEO, psi[k])
        assert np.sqrt(op.norm2(r) / op.norm2(chi[k])) <= 1.05e-10, k
