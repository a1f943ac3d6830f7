"""Orbitals handed over as device pointers: the library copies them and reads its
copies only.  Memory that CUDA does not know is refused before anything touches
it, page-locked host memory is taken as a device pointer, and the context stays
usable after a refusal.  Copies are exact, so energies are equal."""
import ctypes

import numpy as np
import pytest
import torch

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def set_device(ctx, C, eps, o):
    """C column-major; both addresses declared to be device pointers."""
    ptr = lambda x: ctypes.c_void_p(x.data_ptr() if isinstance(x, torch.Tensor) else x.ctypes.data)
    return ctx._lib.mshqc_cd_set_orbitals(ctx._h, capi.ALPHA, ptr(C), ptr(eps), o, capi.DEVICE)


def test_orbital_pointers():
    N, o, M = 24, 5, 60
    inp = syn.make_inputs(N, o, M, seed=8)
    C, eps = np.asfortranarray(inp.alpha.C), np.ascontiguousarray(inp.alpha.eps)
    Ct = torch.from_numpy(np.ascontiguousarray(C.T))
    et = torch.from_numpy(eps)
    with capi.Context(0) as ctx:
        ctx.set_vectors(inp.L).set_orbitals(capi.ALPHA, C, eps, o)
        e = ctx.mp2_energy(capi.RESTRICTED, capi.FP64)["total"]
        assert set_device(ctx, C, et.cuda(), o) == capi.ERR_ARG
        assert set_device(ctx, Ct.cuda(), eps, o) == capi.ERR_ARG
        assert ctx.mp2_energy(capi.RESTRICTED, capi.FP64)["total"] == e
        for c, x in ((Ct.cuda(), et.cuda()), (Ct.pin_memory(), et.pin_memory()), (Ct.cuda(), et.pin_memory())):
            torch.cuda.synchronize()
            assert set_device(ctx, c, x, o) == capi.OK
            assert ctx.mp2_energy(capi.RESTRICTED, capi.FP64)["total"] == e
        bad = et.clone()
        bad[3] = float("nan")
        assert set_device(ctx, Ct.cuda(), bad.cuda(), o) == capi.ERR_NUMERIC
        assert b"eps" in ctx._lib.mshqc_cd_last_error()
