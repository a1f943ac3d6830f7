"""The FP64 path on systems of two distant fragments: vectors that are large on
one fragment are `coupling` times that on the other and between them, in turn,
so the rows of orbitals of different fragments are large in different places
and the integrals between them are far below the product of the row maxima.
Every pair energy and every block of the derivatives is compared with its own
size, which int8 slices alone (held relative to the row maxima) miss by 1e-10
and more.  Tolerances of the FP64 path: 1e-12 relative on energies, 1e-10 of a
block's largest element on derivatives."""
import numpy as np
import pytest

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from oracle import cdmp2_oracle as orc

pytestmark = pytest.mark.gpu


def fragments(n, o, M, coupling, seed, extra=0):
    """Two fragments of n and n + extra functions, o occupied orbitals each."""
    rng = np.random.default_rng(seed)
    N = 2 * n + extra
    side = (np.arange(N) >= n).astype(int)
    L = rng.standard_normal((M, N, N))
    L = 0.05 * (L + L.transpose(0, 2, 1))
    at = np.arange(M) % 2
    big = (side[None, :, None] == at[:, None, None]) & (side[None, None, :] == at[:, None, None])
    L *= np.where(big, 1.0, coupling)
    C = np.zeros((N, N))
    own = np.concatenate([np.repeat([0, 1], o), np.repeat([0, 1], [n - o, n + extra - o])])   # fragment of each orbital
    for f in (0, 1):
        q, _ = np.linalg.qr(rng.standard_normal((np.sum(side == f),) * 2))
        C[np.ix_(side == f, own == f)] = q
    eps = syn.make_orbitals(N, 2 * o, seed).eps
    return L.reshape(M, N * N), C, eps, side, own


@pytest.mark.parametrize("slices", ["on", "off"])
@pytest.mark.parametrize("n,o,M,coupling,extra", [(48, 3, 128, 1e-6, 0), (70, 4, 97, 1e-9, 0), (33, 2, 64, 1e-3, 0),
                                                  (77, 4, 65, 1e-7, 1)])
def test_distant_fragments(monkeypatch, slices, n, o, M, coupling, extra):
    monkeypatch.setenv("MSHQC_CD_FP64_SLICES", slices)
    L, C, eps, side, own = fragments(n, o, M, coupling, n, extra)
    oc = 2 * o
    with capi.Context(0) as ctx:
        ctx.set_vectors(L).set_orbitals(capi.ALPHA, C, eps, oc)
        e = ctx.mp2_energy(capi.RESTRICTED, capi.FP64)["total"]
        pairs = ctx.pair_energies(0)
        g = ctx.mp2_gradient(capi.RESTRICTED, capi.FP64)
    E, pref = orc.rmp2_energy(orc.transform(L, C, oc), eps, oc)
    r = orc.restricted_gradient(L, C, eps, oc)
    assert abs(e - E) <= 1e-12 * abs(E)
    cross = np.abs(pref[:o, o:])
    assert cross.max() < 100 * coupling ** 2 * np.abs(pref).max()
    assert np.max(np.abs(pairs - pref) / np.abs(pref)) <= 1e-12
    assert np.max(np.abs(g.deps_a - r["deps"])) <= 1e-10 * np.max(np.abs(r["deps"]))
    for f in (0, 1):
        for cols in (own == 0, own == 1):
            block = np.ix_(side == f, cols)
            assert np.max(np.abs(g.dC_a - r["dC"])[block]) <= 1e-10 * np.max(np.abs(r["dC"][block]))


def test_fragments_open_shell(monkeypatch):
    monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "on")
    n, o, M, coupling = 40, 3, 80, 1e-7
    L, C, eps, side, own = fragments(n, o, M, coupling, seed=5)
    oa, ob = 2 * o, 2 * o - 1   # beta: the last occupied orbital (fragment 1) is a virtual one
    with capi.Context(0) as ctx:
        ctx.set_vectors(L).set_orbitals(capi.ALPHA, C, eps, oa).set_orbitals(capi.BETA, C, eps, ob)
        ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
        got = [ctx.pair_energies(k) for k in range(3)]
    monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "off")
    with capi.Context(0) as ctx:
        ctx.set_vectors(L).set_orbitals(capi.ALPHA, C, eps, oa).set_orbitals(capi.BETA, C, eps, ob)
        ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
        ref = [ctx.pair_energies(k) for k in range(3)]
    for x, y in zip(got, ref):
        assert np.all(np.abs(x - y) <= 1e-12 * np.abs(y))
