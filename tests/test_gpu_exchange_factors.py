"""Exchange builds through the Cholesky factors of the densities
(mshqc_cd_cholesky_fock): sizes on both sides of the dispatch (N = 96) and of
the tile edges, and densities that must take the full products (full rank,
indefinite, more than N / 4 vectors) alone or beside a factored one.  Against
numpy in FP64, 1e-12 of the largest entry (a sum of about M N^2 products, as
in the other Fock tests)."""
import numpy as np
import pytest

from mshqc_b200 import capi

pytestmark = pytest.mark.gpu


def density(kind, N, rng):
    C, _ = np.linalg.qr(rng.standard_normal((N, N)))
    if kind == "zero":
        return np.zeros((N, N))
    if kind == "full":
        return (C * rng.uniform(0.1, 1.0, N)) @ C.T
    if kind == "indefinite":
        d = np.zeros(N)
        d[:6] = (1.0, -0.7, 0.5, 0.3, -0.2, 0.1)
        return (C * d) @ C.T
    r = {"one": 1, "low": max(2, N // 10), "many": N // 2}[kind]
    return C[:, :r] @ C[:, :r].T


@pytest.mark.parametrize("N,M,kinds", [
    (95, 40, ("low", "low")), (96, 40, ("low", "one")), (97, 33, ("low", "full")), (129, 50, ("indefinite", "low")),
    (128, 50, ("many", "low")), (160, 64, ("zero", "low")), (130, 61, ("low", None)), (130, 61, ("full", None)),
])
def test_factored_exchange(N, M, kinds):
    rng = np.random.default_rng(N + M)
    X = rng.standard_normal((M, N, N)) * 0.05
    L = X + X.transpose(0, 2, 1)
    L[5] *= 1e-9                      # screened out of K in the closed-shell build
    H = rng.standard_normal((N, N))
    H = 0.5 * (H + H.T)
    P = [density(k, N, rng) for k in kinds if k]
    P = [0.5 * (p + p.T) for p in P]
    with capi.Context(0) as ctx:
        ctx.set_vectors(L.reshape(M, N * N))
        out = ctx.cholesky_fock(H, P[0], P[1] if len(P) == 2 else None)
    Ptot = sum(P)
    J = np.einsum("q,qmn->mn", np.einsum("qmn,mn->q", L, Ptot), L)
    keep = [q for q in range(M) if len(P) == 2 or np.linalg.norm(L[q]) > 1e-8]
    close = lambda x, y: np.max(np.abs(x - y)) <= 1e-12 * max(1.0, np.max(np.abs(y)))
    assert close(out["J"], J)
    for p, name in zip(P, "ab"):
        K = sum(L[q] @ p @ L[q] for q in keep)
        assert close(out["K_" + name], K), name
        assert close(out["F_" + name], H + J - (1.0 if len(P) == 2 else 0.5) * K), name
