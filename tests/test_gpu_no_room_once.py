"""Where the memory left holds no slices, a call finds out once and then runs the
FP64 products: as many kernels as with the slices switched off, and one more
where a first operand had been sliced before the second found no room."""
import pytest
import torch

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from test_gpu_slices_no_room import fill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ob", [None, 18])
def test_slices_are_tried_once_a_call(monkeypatch, ob):
    N, oa, M = 203, 20, 601
    inp = syn.make_inputs(N, oa, M, seed=5, nocc_beta=ob)
    kind = capi.RESTRICTED if ob is None else capi.UNRESTRICTED
    torch.cuda.init()

    def launches(ctx):
        ctx.set_orbitals(capi.ALPHA, inp.alpha.C, inp.alpha.eps, oa)
        if ob is not None:
            ctx.set_orbitals(capi.BETA, inp.beta.C, inp.beta.eps, ob)
        at = [ctx.launch_count()]
        for call in (ctx.mp2_energy, ctx.mp2_gradient):
            call(kind, capi.FP64)
            at.append(ctx.launch_count())
        return at[1] - at[0], at[2] - at[1]

    with capi.Context(0) as ctx:
        ctx.set_vectors(inp.L)
        monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "off")
        off = launches(ctx)
        monkeypatch.setenv("MSHQC_CD_FP64_SLICES", "on")
        held = fill(1 << 22)
        try:
            for _ in range(2):
                e, g = launches(ctx)
                assert off[0] <= e <= off[0] + 1 and off[1] <= g <= off[1] + 1
        finally:
            del held
            torch.cuda.empty_cache()
        e, g = launches(ctx)
        assert e > off[0] + 1 and g > off[1] + 1      # with room the slices run
