"""Exchange of a density with parts of very different size: two blocks that the
vectors do not couple, the second `scale` times the first.  Every block of K is
compared with its own largest element, 1e-12 as for K as a whole elsewhere."""
import numpy as np
import pytest

from mshqc_b200 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-8, 1e-16, 1e-20])
@pytest.mark.parametrize("n,o,M", [(64, 8, 40), (61, 5, 33)])
def test_exchange_of_small_blocks(n, o, M, scale):
    rng = np.random.default_rng(n)
    N = 2 * n
    L, P = np.zeros((M, N, N)), np.zeros((N, N))
    for b, s in ((0, 1.0), (1, scale)):
        k = slice(b * n, (b + 1) * n)
        X = rng.standard_normal((M, n, n)) * 0.05
        L[:, k, k] = X + X.transpose(0, 2, 1)
        C, _ = np.linalg.qr(rng.standard_normal((n, n)))
        P[k, k] = s * (C[:, :o] @ C[:, :o].T)
    P = 0.5 * (P + P.T)
    with capi.Context(0) as ctx:
        ctx.set_vectors(L.reshape(M, N * N))
        K = ctx.cholesky_fock(np.eye(N), P)["K_a"]
    for b in (0, 1):
        k = slice(b * n, (b + 1) * n)
        ref = sum(L[q][k, k] @ P[k, k] @ L[q][k, k] for q in range(M))
        assert np.max(np.abs(K[k, k] - ref)) <= 1e-12 * np.max(np.abs(ref)), b
