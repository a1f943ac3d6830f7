"""The sliced FP64 products where the memory left does not hold their slices:
the FP64 products run instead (same bounds: 1e-12 relative on energies, 1e-10
of the largest element on derivatives)."""
import numpy as np
import pytest
import torch

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def fill(keep):
    """Tensors that take the device's free memory down to about `keep` bytes."""
    held, step = [], 1 << 34
    while step >= 1 << 21:
        if torch.cuda.mem_get_info()[0] < keep + step:
            step >>= 1
            continue
        try:
            held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            step >>= 1
    return held


@pytest.mark.parametrize("ob", [None, 18])
def test_fp64_without_room_for_slices(monkeypatch, ob):
    N, oa, M = 203, 20, 601
    inp = syn.make_inputs(N, oa, M, seed=5, nocc_beta=ob)
    ref = capi.RESTRICTED if ob is None else capi.UNRESTRICTED
    torch.cuda.init()

    def run(ctx):
        ctx.set_orbitals(capi.ALPHA, inp.alpha.C, inp.alpha.eps, oa)
        if ob is not None:
            ctx.set_orbitals(capi.BETA, inp.beta.C, inp.beta.eps, ob)
        return ctx.mp2_energy(ref, capi.FP64)["total"], ctx.mp2_gradient(ref, capi.FP64)

    with capi.Context(0) as ctx:
        ctx.set_vectors(inp.L)
        monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "off")
        e0, g0 = run(ctx)
        monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "on")
        held = fill(1 << 22)
        try:
            e1, g1 = run(ctx)
        finally:
            del held
            torch.cuda.empty_cache()
        e2, g2 = run(ctx)
    for e, g in ((e1, g1), (e2, g2)):
        assert abs(e - e0) <= 1e-12 * abs(e0)
        for x, y in zip((g.dC_a, g.deps_a, g.dC_b, g.deps_b), (g0.dC_a, g0.deps_a, g0.dC_b, g0.deps_b)):
            if y is not None:
                assert np.max(np.abs(x - y)) <= 1e-10 * max(1.0, np.max(np.abs(y)))
