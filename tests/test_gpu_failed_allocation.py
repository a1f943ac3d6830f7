"""A call that fails for want of device memory leaves nothing behind that a
later call takes for its own work: with the memory free again the same context
gives the results of a fresh one, without new inputs.  The calls are made to
fail at many places by leaving them between a little and nearly all of the
memory that they ask for.  Bounds of the FP64 and the mixed path: 1e-12 and
1e-9 relative on energies, 1e-10 and 1e-9 of the largest element (at least one)
on derivatives, as elsewhere for the same call with other block sizes."""
import numpy as np
import pytest
import torch

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from test_gpu_slices_no_room import fill

pytestmark = pytest.mark.gpu

N, OA, OB, M = 300, 20, 18, 600


@pytest.fixture(scope="module")
def inp():
    return syn.make_inputs(N, OA, M, seed=13, nocc_beta=OB)


def context(inp, L):
    ctx = capi.Context(0)
    ctx.set_vectors(L)
    ctx.set_orbitals(capi.ALPHA, inp.alpha.C, inp.alpha.eps, OA)
    ctx.set_orbitals(capi.BETA, inp.beta.C, inp.beta.eps, OB)
    return ctx


def retry(inp, call, check):
    """call(ctx) with a share of its memory left; check(results of a retry)."""
    L = torch.from_numpy(inp.L).cuda()
    with context(inp, L) as ctx:
        before = torch.cuda.mem_get_info()[0]
        ref = call(ctx)
        need = before - torch.cuda.mem_get_info()[0]
    failed = 0
    for share in np.geomspace(0.01, 0.9, 24):
        with context(inp, L) as ctx:
            held = fill(int(share * need))
            try:
                call(ctx)
            except capi.CDError as ex:
                assert ex.code == capi.ERR_ALLOC, ex
                failed += 1
            finally:
                del held
                torch.cuda.empty_cache()
            check(call(ctx), ref, share)
    assert failed


def check_energy(e, ref, share):
    for k in ("total", "os", "ss_aa", "ss_bb"):
        assert abs(e[k] - ref[k]) <= 1e-12 * abs(ref["total"]), (share, k)


def check_gradient(e_tol, d_tol):
    def check(g, ref, share):
        assert abs(g.energy["total"] - ref.energy["total"]) <= e_tol * abs(ref.energy["total"]), share
        for x, y in zip((g.dC_a, g.deps_a, g.dC_b, g.deps_b), (ref.dC_a, ref.deps_a, ref.dC_b, ref.deps_b)):
            if y is not None:
                assert np.max(np.abs(x - y)) <= d_tol * max(1.0, np.max(np.abs(y))), share
    return check


@pytest.mark.parametrize("kind", [capi.RESTRICTED, capi.UNRESTRICTED])
def test_energy_after_failed_allocation(inp, kind):
    retry(inp, lambda ctx: ctx.mp2_energy(kind, capi.FP64), check_energy)


@pytest.mark.parametrize("kind", [capi.RESTRICTED, capi.UNRESTRICTED])
@pytest.mark.parametrize("precision", [capi.FP64, capi.FP16X3])
def test_gradient_after_failed_allocation(inp, kind, precision):
    tol = (1e-12, 1e-10) if precision == capi.FP64 else (1e-9, 1e-9)
    retry(inp, lambda ctx: ctx.mp2_gradient(kind, precision), check_gradient(*tol))


def test_complete_vectors_are_kept(inp):
    """MO vectors that an earlier call completed are not formed again after a call
    that fails later: ranks that share a gradient gather them together, and a rank
    that did so alone would wait for the others."""
    L = torch.from_numpy(inp.L).cuda()
    with context(inp, L) as ctx:
        ref = ctx.mp2_gradient(capi.RESTRICTED, capi.FP64)
    with context(inp, L) as ctx:
        ctx.mp2_energy(capi.RESTRICTED, capi.FP64)
        held = fill(8 << 20)
        try:
            with pytest.raises(capi.CDError) as ex:
                ctx.mp2_gradient(capi.RESTRICTED, capi.FP64)
            assert ex.value.code == capi.ERR_ALLOC
        finally:
            del held
            torch.cuda.empty_cache()
        g = ctx.mp2_gradient(capi.RESTRICTED, capi.FP64)
        assert ctx.stage_counts()["transform"] == 0
        check_gradient(1e-12, 1e-10)(g, ref, 1.0)
