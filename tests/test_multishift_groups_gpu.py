"""Mixed-precision multi-shift solves with more shifts than the context's max_rhs: the FP64 refinement runs in
groups of max_rhs shifts (whole groups, a last group of one, one shift per group).  Every shift by the
oracle's FP64 residual, with the tolerance of test_multishift_gpu.py."""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [G.PREC_SINGLE, G.PREC_HALF], ids=["f32", "f16"])
@pytest.mark.parametrize("max_rhs,ns", [(2, 4), (2, 5), (1, 3), (12, 13)])
def test_more_shifts_than_right_hand_sides(max_rhs, ns, prec):
    from oracle import Oracle, OracleOp
    from oracle import oracle as O
    dims, mass, csw = (4, 4, 4, 8), 1 / (2 * 0.115) - 4, 1.0
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 31), (1, 1, 1, -1))
    op = OracleOp(dims, u, mass, csw)
    chi = S.z2_noise(dims, 14, cb=1).reshape(-1, 12)
    shifts = [0.0] + [0.01 * 2.0 ** k for k in range(ns - 1)]
    ctx = G.Context(dims, mass, csw, t_boundary=-1, max_rhs=max_rhs)
    try:
        ctx.load_gauge(u)
        psi, res, rc = ctx.solve_multishift(chi, shifts, rsd_target=1e-10, sloppy_precision=prec)
    finally:
        ctx.close()
    assert rc == 0, res
    for k, sigma in enumerate(shifts):
        r = chi - op.apply(O.OP_MDAGM, psi[k]) - sigma * psi[k]
        rel = np.sqrt(op.norm2(r) / op.norm2(chi))
        assert rel <= 1.5e-10, (sigma, res[k])
        assert abs(res[k]["rel_resid"] - rel) <= 1e-12
