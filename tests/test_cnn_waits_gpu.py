"""A network layer's wait for the tensor cores that gives up fails the call whichever warp it happens in:
the warp that issues the MMA (0), one that only stores (2), one that only gathers (8).  GBC_TC_QUIT_WARP makes
the waits of one warp give up at once; the block then waits for its MMA all the same and leaves.

Exact: a call either fails, or its result is the one of an undisturbed network."""
import threading

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu

MASS, CSW = 1 / (2 * 0.115) - 4, 1.0


def _context(dims, max_rhs=2):
    ctx = G.Context(dims, MASS, CSW, t_boundary=-1, max_rhs=max_rhs)
    ctx.load_gauge(G.gauge_synthetic(dims, 0.3, 5, t_boundary=-1))
    return ctx


@pytest.mark.parametrize("warp", [0, 2, 8])
@pytest.mark.parametrize("dims,nrhs", [((4, 4, 4, 4), 1),       # one MMA per block: nothing follows the wait
                                       ((16, 16, 16, 16), 2)])  # blocks that walk several tiles
def test_given_up_wait_fails_the_call(dims, nrhs, warp, monkeypatch):
    x = np.stack([S.gaussian(dims, 30 + k, cb=1).reshape(-1, 12) for k in range(nrhs)]).astype(np.complex128)
    ctx = _context(dims)
    try:
        ctx.precond_init(hidden=12, layers=3, seed=1)
        want = ctx.precond_apply(x)
        monkeypatch.setenv("GBC_TC_QUIT_WARP", str(warp))
        ctx.precond_init(hidden=12, layers=3, seed=1)
        monkeypatch.delenv("GBC_TC_QUIT_WARP")
        for call in (lambda: ctx.precond_apply(x), lambda: ctx.precond_loss_grad(x, x),
                     lambda: ctx.solve(x[:1], solver=G.SOLVER_FGMRES, use_precond=1)):
            with pytest.raises(G.GBCError, match="tensor cores"):
                call()
        ctx.precond_init(hidden=12, layers=3, seed=1)
        assert np.array_equal(ctx.precond_apply(x), want)
    finally:
        ctx.close()


def test_contexts_count_their_own_waits(monkeypatch):
    """Two contexts on two threads, the waits of one giving up: each of its calls fails, and none of the calls
    that the other makes meanwhile."""
    x = S.gaussian((8, 8, 8, 8), 3, cb=1).reshape(1, -1, 12).astype(np.complex128)
    y = S.gaussian((16, 16, 16, 16), 3, cb=1).reshape(1, -1, 12).astype(np.complex128)
    bad, good = _context((16, 16, 16, 16)), _context((8, 8, 8, 8))
    try:
        good.precond_init(hidden=12, layers=2, seed=1)
        want = good.precond_apply(x)
        monkeypatch.setenv("GBC_TC_QUIT_WARP", "0")
        bad.precond_init(hidden=12, layers=8, seed=1)
        monkeypatch.delenv("GBC_TC_QUIT_WARP")
        failed, right, done = [], [], threading.Event()

        def fails():
            for _ in range(100):
                try:
                    bad.precond_apply(y)
                    failed.append(False)
                except G.GBCError:
                    failed.append(True)
            done.set()

        def works():
            while not done.is_set():
                try:
                    right.append(np.array_equal(good.precond_apply(x), want))
                except G.GBCError:
                    right.append(False)

        threads = [threading.Thread(target=f) for f in (fails, works)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert all(failed) and all(right) and len(right) > 1
    finally:
        bad.close()
        good.close()
