"""Separate contexts are independent: solves of two contexts on two threads at once (each with its helper
thread for the result pages, its copy stream and its captured iterations), operator and network calls
between them, give bit for bit what the same calls give one after the other.

Launch shapes come from a tune cache that the first, sequential run fills: another shape would sum in
another order."""
import threading

import numpy as np
import pytest

from chroma_gb300 import gbclover as G
from chroma_gb300 import sources as S

pytestmark = pytest.mark.gpu


def _calls(dims, seed, nrhs):
    """Everything one thread does: its own context, from creation to its last call."""
    out = []
    ctx = G.Context(dims, 1 / (2 * 0.115) - 4, 1.0, t_boundary=-1, max_rhs=nrhs)
    try:
        ctx.load_gauge(G.gauge_synthetic(dims, 0.3, seed, t_boundary=-1))
        chi = np.stack([S.z2_noise(dims, seed + k, cb=1).reshape(-1, 12) for k in range(nrhs)])
        ctx.precond_init(hidden=12, layers=2, seed=seed)
        for _ in range(3):
            for solver, system in ((G.SOLVER_BICGSTAB, G.SYS_FULL), (G.SOLVER_MIXED, G.SYS_MEO), (G.SOLVER_CG, G.SYS_MEO),
                                   (G.SOLVER_BICGSTAB, G.SYS_SYM)):
                psi, _, rc = ctx.solve(chi, solver=solver, system=system, rsd_target=1e-9, delta=0.05)
                assert rc == 0
                out.append(psi)
            out.append(ctx.solve_multishift(chi[0], [0.01, 0.3], sloppy_precision=G.PREC_SINGLE)[0])
            out.append(ctx.precond_apply(chi))
            out.append(ctx.apply(G.OP_MEO, chi, 1, 1, G.PREC_DOUBLE))
    finally:
        ctx.close()
    return out


def test_two_contexts_on_two_threads(tmp_path, monkeypatch):
    monkeypatch.setenv("GBC_TUNE_CACHE", str(tmp_path / "tune.cache"))
    jobs = [((8, 8, 8, 16), 3, 2), ((8, 6, 8, 12), 40, 3)]
    _ = [_calls(*j) for j in jobs]  # fills the cache
    want = [_calls(*j) for j in jobs]
    got, errors = [None, None], []

    def run(k):
        try:
            got[k] = _calls(*jobs[k])
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert len(got[k]) == len(want[k])
        for i, (a, b) in enumerate(zip(got[k], want[k])):
            assert np.array_equal(a, b), (k, i)
