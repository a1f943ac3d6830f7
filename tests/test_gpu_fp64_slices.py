"""The FP64 path through int8 slices of full accuracy (ozaki_i8.cuh, Full),
forced at sizes around its tile edges (128 rows, 64 columns, 32-wide K chunks,
64-wide virtual padding) against the oracle, and at a size where the dispatch
itself takes it.  Tolerances of the FP64 path: 1e-12 relative on energies,
1e-10 of the largest element on derivatives (derived for FP64 products; the
slices' error per term is below 2^-55 of the row maxima)."""
import os

import numpy as np
import pytest

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from oracle import cdmp2_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture
def slices(monkeypatch):
    monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "on")


def close(x, y, tol=1e-10):
    return np.max(np.abs(x - y)) <= tol * max(1.0, np.max(np.abs(y)))


def check(N, oa, ob, M, seed):
    inp = syn.make_inputs(N, oa, M, seed=seed, nocc_beta=ob)
    a, b = inp.alpha, inp.beta
    with capi.Context(0) as ctx:
        ctx.set_vectors(inp.L).set_orbitals(capi.ALPHA, a.C, a.eps, oa)
        if ob is None:
            e = ctx.mp2_energy(capi.RESTRICTED, capi.FP64)
            pairs = ctx.pair_energies(0)
            g = ctx.mp2_gradient(capi.RESTRICTED, capi.FP64)
            E, pref = orc.rmp2_energy(orc.transform(inp.L, a.C, oa), a.eps, oa)
            r = orc.restricted_gradient(inp.L, a.C, a.eps, oa)
            assert abs(e["total"] - E) <= 1e-12 * abs(E)
            assert np.max(np.abs(pairs - pref)) <= 1e-12 * np.max(np.abs(pref))
            assert abs(g.energy["total"] - r["E"]) <= 1e-12 * abs(r["E"])
            assert close(g.dC_a, r["dC"]) and close(g.deps_a, r["deps"])
        else:
            ctx.set_orbitals(capi.BETA, b.C, b.eps, ob)
            e = ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
            g = ctx.mp2_gradient(capi.UNRESTRICTED, capi.FP64)
            r = orc.unrestricted_gradient(inp.L, a.C, b.C, a.eps, b.eps, oa, ob)
            for k in ("ss_aa", "ss_bb", "os"):
                assert abs(e[k] - r[k]) <= 1e-12 * max(abs(r[k]), 1e-3 * abs(r["E"])), k
            assert abs(g.energy["total"] - r["E"]) <= 1e-12 * abs(r["E"])
            assert close(g.dC_a, r["dC_a"]) and close(g.dC_b, r["dC_b"])
            assert close(g.deps_a, r["deps_a"]) and close(g.deps_b, r["deps_b"])


@pytest.mark.parametrize("N,oa,ob,M", [
    (20, 2, None, 17), (66, 2, None, 32), (67, 3, None, 33), (131, 2, None, 95), (72, 8, 7, 64), (70, 5, 1, 129),
])
@pytest.mark.parametrize("block", [None, 2])
def test_sliced_fp64_vs_oracle(slices, monkeypatch, N, oa, ob, M, block):
    if block:
        monkeypatch.setenv("MSHQC_CD_BWD_BLOCK", str(block))
    check(N, oa, ob, M, seed=N + M)


def test_dispatched_size_vs_oracle():
    assert "MSHQC_CD_FP64_SLICES" not in os.environ
    check(203, 20, None, 601, seed=5)


def test_long_k_segments(slices):
    """Gamma over more columns (400 x 64) than one exact accumulation holds."""
    check(430, 400, None, 40, seed=9)


def test_row_with_wide_range(slices):
    """Vectors over 200 orders of magnitude: rows far below and above one."""
    N, o, M = 40, 4, 48
    inp = syn.make_inputs(N, o, M, seed=2)
    L = inp.L * np.ldexp(1.0, np.linspace(-300, 60, M).astype(int))[:, None]
    a = inp.alpha
    with capi.Context(0) as ctx:
        ctx.set_vectors(L).set_orbitals(capi.ALPHA, a.C, a.eps, o)
        B = ctx.transform(capi.ALPHA, capi.FP64)
        e = ctx.mp2_energy(capi.RESTRICTED, capi.FP64)["total"]
    Br = orc.transform(L, a.C, o)
    # each vector's column is relative to its own scale: K of the transform is nu
    scale = np.max(np.abs(Br), axis=(0, 1), keepdims=True)
    assert np.max(np.abs(B - Br) / scale) <= 1e-13
    E, _ = orc.rmp2_energy(Br, a.eps, o)
    assert abs(e - E) <= 1e-12 * abs(E)
