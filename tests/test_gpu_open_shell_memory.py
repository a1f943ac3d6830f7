"""Open-shell calls in the memory that one spin's half-transformed vectors at a
time leave them: the MO vectors of both spins, the larger Y and, for the
gradient, both Gamma and the smallest staging (one row orbital against all
columns, integrals and amplitudes), and 40 MB for everything small (with 24 the
staging, which takes what it finds, leaves the gradient's per-pair sums none).  Results as
with plenty of memory, 1e-12 relative (energies) and 1e-10 of the largest
element (derivatives)."""
import numpy as np
import pytest
import torch

from mshqc_b200 import capi
from mshqc_b200 import synthetic as syn
from test_gpu_slices_no_room import fill

pytestmark = pytest.mark.gpu

N, OA, OB, M = 420, 30, 29, 700


def context(inp, L):
    ctx = capi.Context(0)
    ctx.set_vectors(L)
    ctx.set_orbitals(capi.ALPHA, inp.alpha.C, inp.alpha.eps, OA)
    ctx.set_orbitals(capi.BETA, inp.beta.C, inp.beta.eps, OB)
    return ctx


def test_open_shell_with_one_spin_at_a_time():
    inp = syn.make_inputs(N, OA, M, seed=1, nocc_beta=OB)
    L = torch.from_numpy(inp.L).cuda()
    vp, Mp = -(-(N - OB) // 64) * 64, -(-M // 16) * 16
    B, Y = 8 * (OA + OB) * vp * Mp, 8 * OA * M * N
    staging = 16 * vp * OB * vp
    spare = 40 << 20
    with context(inp, L) as ctx:
        e0 = ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
        g0 = ctx.mp2_gradient(capi.UNRESTRICTED, capi.FP64)
    for room in (B + Y + spare, 2 * B + Y + staging + spare):
        with context(inp, L) as ctx:
            held = fill(room)
            try:
                if room < 2 * B:
                    e = ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
                    e2 = ctx.mp2_energy(capi.UNRESTRICTED, capi.FP64)
                else:
                    g = ctx.mp2_gradient(capi.UNRESTRICTED, capi.FP64)
            finally:
                del held
                torch.cuda.empty_cache()
    for x in (e, e2, g.energy):
        assert abs(x["total"] - e0["total"]) <= 1e-12 * abs(e0["total"])
    for x, y in zip((g.dC_a, g.deps_a, g.dC_b, g.deps_b), (g0.dC_a, g0.deps_a, g0.dC_b, g0.deps_b)):
        assert np.max(np.abs(x - y)) <= 1e-10 * np.max(np.abs(y))
