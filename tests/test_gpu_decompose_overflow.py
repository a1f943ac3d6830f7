"""A decomposition whose numbers overflow on the way: one CTA's diagonals are all
NaN from some step on and it has no candidate for the pivot.  N = 6: 36
elements, 32 in the first CTA.  Its elements overflow in step 0 (1.7e308 over a
pivot of 0.1) and turn to NaN in step 1 (infinity times zero); the pivots lie in
the second CTA.  Operations in the order of the kernel, so equal to the bit."""
import numpy as np
import pytest

from mshqc_b200 import capi

pytestmark = pytest.mark.gpu


def decompose(E, thr):
    """The reference's loop; a NaN is never larger than anything."""
    D, L = np.diag(E).copy(), []
    with np.errstate(all="ignore"):
        while len(L) < len(D):
            p, best = 0, -np.inf
            for k, d in enumerate(D):
                if d > best:
                    p, best = k, d
            if best < thr:
                break
            col = E[:, p].copy()
            for l in L:
                col = col - l * l[p]
            nf = np.sqrt(best)
            L.append(col / nf if nf > 1e-12 else col)
            D = D - L[-1] * L[-1]
            D[D < 0.0] = 0.0
    return np.array(L)


def test_cta_without_a_candidate():
    n = 36
    E = np.diag(np.full(n, 1e-3))
    for step, p in enumerate((33, 35, 32, 34)):
        E[p, p] = 1e-2 / (step + 1)
    E[:32, 33] = E[33, :32] = 1.7e308
    ref = decompose(E, 1e-6)
    assert len(ref) == 4 and np.isnan(ref[1, :32]).all()
    with capi.Context(0) as c:
        L = c.cholesky_decompose(E.reshape(6, 6, 6, 6), 1e-6)
        assert np.array_equal(L, ref, equal_nan=True)
        E2 = np.diag(np.full(n, 1e-3))   # the context goes on
        assert np.array_equal(c.cholesky_decompose(E2.reshape(6, 6, 6, 6), 1e-6), decompose(E2, 1e-6))
