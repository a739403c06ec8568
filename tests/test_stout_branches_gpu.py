"""Stout smearing at the edges of its kernel: lattices whose site count is below, at and not a
multiple of a block's 32 sites, and weights that take exp(iQ) through each of its ranges of
c1 = tr(Q^2)/2 (12 Taylor terms below 0.05, 20 below 0.75, the closed form above).

The oracle runs the same formulas in FP64: 1e-12, as in test_stout_gpu.py."""
import numpy as np
import pytest

from chroma_gb300 import gbclover as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,eps,rho,lo,hi", [
    ((2, 2, 2, 2), 0.2, 0.02, 0.0, 0.05),
    ((4, 2, 4, 2), 0.3, 0.08, 0.0, 0.75),
    ((2, 6, 2, 4), 1.0, 0.2, 0.05, 8.0),
    ((6, 2, 6, 2), 1.5, 0.6, 0.75, 60.0),
])
def test_ranges_match_oracle(dims, eps, rho, lo, hi):
    from oracle import Oracle
    o = Oracle()
    u = o.gauge_hot(dims, eps, 5)
    want = o.stout(dims, u, rho, 1)
    # c1 of the exponents the step applied: exp(iQ) = U' U^dag, with eigenvalues exp(i lambda)
    e = np.einsum("vmij,vmkj->vmik", want, u.conj())
    if rho < 0.3:  # |lambda| < pi: the angles are the eigenvalues of Q
        c1 = 0.5 * (np.angle(np.linalg.eigvals(e)) ** 2).sum(-1)
        assert c1.min() < hi and c1.max() > lo
    got = G.stout_smear(dims, u, 1, rho)
    assert np.max(np.abs(got - want)) < 1e-12
