"""The FP64 one-thread-per-site stencil (hop_kernel), which serves lattices above the split kernel's limit, on
small lattices with its launch shapes pinned (GBC_SHAPE): ragged last blocks, partly filled right-hand-side
groups, both isigns, every epilogue, the twisted-mass terms and the reductions of CG and BiCGStab.

Against the CPU oracle: operators 1e-12 relative, as the FP64 operators of test_gpu_parity.py; solutions by the
oracle's FP64 residual.  The tune report says which launches ran on the pinned shape."""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.1
# the shapes that take FP64, by their index in kHopShapes: sites x right-hand sides (resident blocks)
SHAPES = {0: "tx=128 nrb=1 minb=1", 1: "tx=128 nrb=1 minb=6", 2: "tx=32 nrb=4 minb=1", 3: "tx=32 nrb=4 minb=5",
          4: "tx=64 nrb=2 minb=4", 5: "tx=32 nrb=12 minb=2"}
NRB = {0: 1, 1: 1, 2: 4, 3: 4, 4: 2, 5: 12}
CASES = [(s, n) for s in SHAPES for n in (1, 5, 12) if NRB[s] <= n]


def _setup(dims, twisted_m=None):
    from oracle import Oracle, OracleOp
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 99), (1, 1, 1, -1))
    return u, OracleOp(dims, u, MASS, CSW, twisted_m=twisted_m)


def _pinned(ctx, shape):
    """(mode, reduce) of the FP64 launches that ran on the pinned shape; nothing else may have been tuned."""
    out = set()
    for line in ctx.tune_report().strip().splitlines():
        f = dict(w.split("=") for w in line.split(" -> ")[0].split())
        if f["prec"] == "8":
            assert SHAPES[shape] in line and "(GBC_SHAPE)" in line, line
            out.add((int(f["mode"]), int(f["reduce"])))
    return out


@pytest.mark.parametrize("shape,nrhs", CASES)
@pytest.mark.parametrize("dims,mu", [((2, 2, 2, 6), None), ((6, 6, 6, 10), 0.07)], ids=["2x2x2x6", "6x6x6x10-twisted"])
def test_operators(dims, mu, shape, nrhs, monkeypatch):
    from oracle import oracle as O
    monkeypatch.setenv("GBC_SHAPE", str(shape))
    u, op = _setup(dims, mu)
    V = int(np.prod(dims))
    par = S.parity(dims)
    xs = np.stack([S.gaussian(dims, 300 + k).reshape(V, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs, twisted_m=mu)
    try:
        ctx.load_gauge(u)
        for gop, oop, cb in ((G.OP_DSLASH, O.OP_DSLASH, 0), (G.OP_DSLASH, O.OP_DSLASH, 1), (G.OP_MEO, O.OP_MEO, 1),
                             (G.OP_SYM, O.OP_SYM, 1)):
            for isign in (1, -1):
                got = ctx.apply(gop, xs, isign, cb, G.PREC_DOUBLE)
                for k in {0, nrhs - 1}:
                    want = op.apply(oop, xs[k], isign, cb)[par == cb]
                    assert np.linalg.norm(got[k][par == cb] - want) < 1e-12 * np.linalg.norm(want), (gop, cb, isign, k)
        # plain, clover, xpay and (not compiled for shape 2) the symmetric operator's second step
        assert {m for m, _ in _pinned(ctx, shape)} == {0, 1, 2, 3} - ({3} if shape == 2 else set())
    finally:
        ctx.close()


@pytest.mark.parametrize("shape,nrhs", CASES)
@pytest.mark.parametrize("solver,system,ends", [(G.SOLVER_CG, G.SYS_MEO, (2, 1)), (G.SOLVER_BICGSTAB, G.SYS_MEO, (2, 2)),
                                                (G.SOLVER_CG, G.SYS_SYM, (3, 1)), (G.SOLVER_BICGSTAB, G.SYS_SYM, (3, 2))],
                         ids=["cg", "bicgstab", "cg-sym", "bicgstab-sym"])
def test_reductions_in_solves(solver, system, ends, shape, nrhs, monkeypatch):
    from oracle import oracle as O
    dims = (6, 4, 6, 10)
    monkeypatch.setenv("GBC_SHAPE", str(shape))
    u, op = _setup(dims)
    chi = np.stack([S.z2_noise(dims, 7 + k, cb=1).reshape(-1, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs, sloppy_precision=G.PREC_DOUBLE)
    try:
        ctx.load_gauge(u)
        psi, res, rc = ctx.solve(chi, solver=solver, system=system, rsd_target=1e-11, sloppy_precision=G.PREC_DOUBLE)
        ran = _pinned(ctx, shape)
    finally:
        ctx.close()
    assert rc == 0
    assert ends in ran or (shape == 2 and system == G.SYS_SYM)  # the reduction in the stencil's epilogue
    oop = O.OP_SYM if system == G.SYS_SYM else O.OP_MEO
    for k in range(nrhs):
        r = chi[k] - op.apply(oop, psi[k])
        assert np.sqrt(op.norm2(r) / op.norm2(chi[k])) <= 1.05e-11, k
