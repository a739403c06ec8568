"""Layer and weight-gradient kernels of the network at the edges of their tiles: 32 sites of one
parity per tile (lattices with fewer sites than a tile, with a ragged last tile and with whole
tiles), every compiled layer shape, and one or several right-hand sides.

Reference: oracle/cnn.py.  Tolerances as in test_cnn_gpu.py: BF16 operands with FP32 sums give
2e-2 on outputs and 5e-2 on gradients (relative norms).
"""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


@pytest.mark.parametrize("dims,hidden,layers,nrhs", [
    ((2, 2, 2, 2), 12, 4, 1),      # 8 sites per parity: a quarter of a tile, wrap-around neighbours
    ((2, 2, 2, 6), 12, 3, 2),      # 24 sites
    ((4, 4, 2, 4), 4, 4, 3),       # 64 sites: two whole tiles, 4 -> 4 layers
    ((6, 4, 2, 6), 12, 2, 5),      # 144 sites: a half-filled last tile, no 12 -> 12 layer
    ((4, 2, 6, 6), 4, 1, 1),       # one layer: odd input and odd output only
    ((6, 6, 6, 10), 12, 4, 13),    # 1080 sites: a ragged last tile, an odd batch spread over blocks
])
def test_tiles_match_oracle(dims, hidden, layers, nrhs):
    from oracle import Oracle
    from oracle.cnn import CnnOracle
    o = Oracle()
    u = o.apply_bc(dims, o.gauge_hot(dims, 0.3, 7), (1, 1, 1, -1))
    V = int(np.prod(dims))
    ctx = G.Context(dims, 1 / (2 * 0.12) - 4, 1.0, t_boundary=-1, max_rhs=16)
    try:
        ctx.load_gauge(u)
        ctx.precond_init(hidden=hidden, layers=layers, seed=11)
        rng = np.random.default_rng(3)
        w = ctx.precond_weights()
        w = w + 0.05 * rng.standard_normal(w.size).astype(np.float32)
        ctx.precond_set_weights(w)
        Ws, k, z = [], 0, w[0::2] + 1j * w[1::2]
        for l in range(layers):
            ci, co = 4 if l == 0 else hidden, 4 if l == layers - 1 else hidden
            Ws.append(z[k:k + 9 * co * ci].reshape(9, co, ci))
            k += 9 * co * ci
        net = CnnOracle(dims, u)
        xs = np.stack([S.gaussian(dims, 50 + b, cb=1).reshape(V, 12) for b in range(nrhs)])
        es = np.stack([S.gaussian(dims, 80 + b, cb=1).reshape(V, 12) for b in range(nrhs)])
        got = ctx.precond_apply(xs)
        for b in range(nrhs):
            assert _rel(got[b], net.apply(xs[b], Ws).reshape(V, 12)) < 2e-2, b
        assert np.all(got[:, S.parity(dims) == 0] == 0)
        loss, g = ctx.precond_loss_grad(xs, es)
        oloss, og = net.loss_grad(list(xs), list(es), Ws)
        assert abs(loss - oloss) < 2e-2 * oloss
        assert _rel(g[0::2] + 1j * g[1::2], np.concatenate([x.reshape(-1) for x in og])) < 5e-2
    finally:
        ctx.close()
