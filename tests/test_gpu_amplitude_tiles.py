"""The backward's amplitude pass at the edges of its 32 x 32 tiles (virtuals
just below, at and above one, two and three tiles), for the modes whose
mirrored tiles go together and the one whose tiles go alone, with and without
mirrored block pairs.  Tolerances of the two paths: FP64 1e-10 of the largest
element against the oracle; mixed 1e-6 on scaled-twin inputs."""
import numpy as np
import pytest

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from oracle import cdmp2_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [None, "2"])
@pytest.mark.parametrize("v", [1, 31, 32, 33, 64, 65, 97])
def test_amplitude_tiles_vs_oracle(monkeypatch, v, block):
    oa, ob = 5, 3
    N, M = v + oa, 2 * (v + oa)
    if block:
        monkeypatch.setenv("MSHQC_CD_BWD_BLOCK", block)
    base = syn.make_inputs(N, oa, M, seed=v, nocc_beta=ob)
    inp = syn.make_inputs(N, oa, M, seed=v, nocc_beta=ob, sigma=syn.twin_sigma(N, oa, M, base.alpha.eps))
    a, b = inp.alpha, inp.beta
    r = orc.restricted_gradient(inp.L, a.C, a.eps, oa)
    u = orc.unrestricted_gradient(inp.L, a.C, b.C, a.eps, b.eps, oa, ob)
    with capi.Context(0) as ctx:
        for prec in (capi.FP64, capi.FP16X3):
            ctx.set_vectors(inp.L).set_orbitals(capi.ALPHA, a.C, a.eps, oa)
            ctx.set_orbitals(capi.BETA, b.C, b.eps, ob)
            g = ctx.mp2_gradient(capi.RESTRICTED, prec)
            h = ctx.mp2_gradient(capi.UNRESTRICTED, prec)
            for x, y in ((g.dC_a, r["dC"]), (g.deps_a, r["deps"]), (h.dC_a, u["dC_a"]), (h.dC_b, u["dC_b"]),
                         (h.deps_a, u["deps_a"]), (h.deps_b, u["deps_b"])):
                tol = 1e-10 * max(1.0, np.max(np.abs(y))) if prec == capi.FP64 else 1e-6
                assert np.max(np.abs(x - y)) <= tol
            for x, y in ((g.energy["total"], r["E"]), (h.energy["total"], u["E"])):
                assert abs(x - y) <= (1e-12 * abs(y) if prec == capi.FP64 else 1e-6)
