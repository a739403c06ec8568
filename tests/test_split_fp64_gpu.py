"""The FP64 stencil whose hops are split over threads, at the edges of its blocks (8, 16 or 32 sites of
one right-hand side): fewer sites than a block, ragged last blocks, extents of 2 where both neighbours
coincide, and the block size each number of right-hand sides selects; both isigns, every epilogue, the
reductions of CG and BiCGStab, and the no-allocation entry point with its output on its input.

Against the CPU oracle: 1e-12 relative, as the FP64 operators of test_gpu_parity.py."""
import ctypes as C

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.1


def _rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def _setup(dims):
    from oracle import Oracle, OracleOp
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 99), (1, 1, 1, -1))
    return u, OracleOp(dims, u, MASS, CSW)


@pytest.mark.parametrize("dims,nrhs", [
    ((2, 2, 2, 2), 1),      # 8 sites: one block
    ((2, 6, 2, 6), 3),      # 72 sites: blocks of 8
    ((6, 6, 6, 10), 12),    # 1080 sites x 12: blocks of 16, the last half full
    ((6, 6, 10, 10), 12),   # 1800 sites x 12: blocks of 32, the last with 8 sites
])
def test_operators(dims, nrhs):
    from oracle import oracle as O
    u, op = _setup(dims)
    V = int(np.prod(dims))
    par = S.parity(dims)
    xs = np.stack([S.gaussian(dims, 300 + k).reshape(V, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs)
    try:
        ctx.load_gauge(u)
        for gop, oop, cbs in ((G.OP_DSLASH, O.OP_DSLASH, (0, 1)), (G.OP_MEO, O.OP_MEO, (1,)),
                              (G.OP_UNPREC, O.OP_UNPREC, (1,))):
            for cb in cbs:
                for isign in (1, -1):
                    got = ctx.apply(gop, xs, isign, cb, G.PREC_DOUBLE)
                    sel = np.ones(V, bool) if gop == G.OP_UNPREC else par == cb
                    for k in (0, nrhs - 1):
                        want = op.apply(oop, xs[k], isign, cb)
                        assert _rel(got[k][sel], want[sel]) < 1e-12, (gop, cb, isign, k)
    finally:
        ctx.close()


@pytest.mark.parametrize("solver", [G.SOLVER_CG, G.SOLVER_BICGSTAB], ids=["cg", "bicgstab"])
@pytest.mark.parametrize("dims,nrhs", [((4, 2, 6, 6), 1), ((6, 6, 6, 10), 12)])
def test_reductions_in_solves(dims, nrhs, solver):
    from oracle import oracle as O
    u, op = _setup(dims)
    chi = np.stack([S.z2_noise(dims, 7 + k, cb=1).reshape(-1, 12) for k in range(nrhs)])
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=nrhs, sloppy_precision=G.PREC_DOUBLE)
    try:
        ctx.load_gauge(u)
        psi, res, rc = ctx.solve(chi, solver=solver, rsd_target=1e-11, sloppy_precision=G.PREC_DOUBLE)
    finally:
        ctx.close()
    assert rc == 0
    for k in range(nrhs):
        r = chi[k] - op.apply(O.OP_MEO, psi[k])
        assert np.sqrt(op.norm2(r) / op.norm2(chi[k])) <= 1.05e-11


@pytest.mark.parametrize("isign", [1, -1])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 6, 2, 6), (6, 6, 10, 10)])
def test_noalloc_in_place(dims, isign):
    import torch
    from oracle import oracle as O
    u, op = _setup(dims)
    V = int(np.prod(dims))
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=1)
    try:
        ctx.load_gauge(u)
        clov, inv, _, _ = ctx.get_clover()
    finally:
        ctx.close()
    x = S.gaussian(dims, 4).reshape(V, 12)
    links = torch.from_numpy(np.ascontiguousarray(u)).cuda()
    tc, ti = torch.from_numpy(clov).cuda(), torch.from_numpy(inv).cuda()
    f = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    lib = G.load()
    geom = G.Geom((C.c_int * 4)(*dims), -1)
    act = G.Action(MASS, CSW, CSW, 0, 1.0, 1.0, 3, 0, 0.0)
    fn = lib.gbc_apply_meo_noalloc
    fn.argtypes = [C.POINTER(G.Geom), C.POINTER(G.Action)] + [C.c_void_p] * 3 + [C.c_int] + [C.c_void_p] * 3
    torch.cuda.synchronize()
    rc = fn(C.byref(geom), C.byref(act), links.data_ptr(), tc.data_ptr(), ti.data_ptr(), isign, f.data_ptr(),
            f.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    odd = S.parity(dims) == 1
    got = f.cpu().numpy()
    assert _rel(got[odd], op.apply(O.OP_MEO, x, isign)[odd]) < 1e-12
    assert np.array_equal(got[~odd], x[~odd])
