"""The one-kernel decomposition at sizes around its work split (32 elements per
CTA, one CTA; ragged last CTA; more vectors than one staged piece of the pivot
row; full rank, where it ends after N^2 vectors).  Same operations in the same
order as the oracle, so 1e-12 of the largest element (the oracle may contract
nothing)."""
import numpy as np
import pytest

from mshqc_b200 import capi
from oracle import cdmp2_oracle as orc

pytestmark = pytest.mark.gpu


def eri(N, rank, seed, full=False):
    rng = np.random.default_rng(seed)
    if full:                                  # positive definite on all N^2 elements
        A = rng.standard_normal((N * N, N * N))
        return (A @ A.T / (N * N) + np.eye(N * N)).reshape(N, N, N, N)
    X = rng.standard_normal((rank, N, N))
    A = (0.2 * (X + X.transpose(0, 2, 1)) * 10.0 ** (-np.arange(rank) / rank)[:, None, None]).reshape(rank, N * N)
    return (A.T @ A).reshape(N, N, N, N)


@pytest.mark.parametrize("N,rank,full", [(2, 2, False), (5, 9, False), (6, 12, False), (9, 30, False), (17, 80, False),
                                         (48, 1060, False), (6, 0, True)])
def test_decompose_split(N, rank, full):
    E = eri(N, rank, 100 * N + rank, full)
    ref = orc.cholesky_decompose(E, 1e-6)
    with capi.Context(0) as c:
        L = c.cholesky_decompose(E, 1e-6)
        assert c.decompose_converged == (not full)
    assert L.shape == ref.shape
    assert np.max(np.abs(L - ref)) <= 1e-12 * max(1.0, np.max(np.abs(ref)))
