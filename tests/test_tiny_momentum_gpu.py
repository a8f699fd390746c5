"""Momentum advection of a component that is rounding alone: small against everything else, down to 1e-24.

The advected momentum is homogeneous of degree 1 in the momentum (every limiter is), so that a component scaled by a
power of two gives the same result scaled by it.  FP32 pairs hold 46 bits of values of this size, and a flux is some ten
operations: 1e-12 of the largest value.
"""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr

pytestmark = pytest.mark.gpu
LIMITERS = ["Koren", "minmod", "vanAlbada1", "Sweby", "superbee", "TVDcen", "TVDdown"]


def advected(limiter, arith, scale, D):
    dims = (22, 18, 14)[:D]
    sim = ia.TwoPhaseSimulation(dims, (0.0,) * D, 14.0, poisson="mixed", λ=limiter, momentum_arith=arith, λρ=0.05,
                                InterfaceSDF=lambda x: torch.sqrt(sum((v - 8.0) ** 2 for v in x)) - 4.0)
    gen = torch.Generator(device="cuda").manual_seed(3)
    u, rhou, old = (fzeros(tuple(sim.flow.u.shape)) for _ in range(3))
    for t in (u, rhou, old):
        t.copy_(0.1 * torch.rand(t.shape, generator=gen, dtype=torch.float64, device="cuda") - 0.05)
    for d in range(D):          # walls
        u[..., d].narrow(d, 0, 2).zero_()
        u[..., d].narrow(d, dims[d] + 1, 1).zero_()
    for t in (rhou, old):
        t[..., D - 1] *= scale
    sim.intf.rhou.copy_(rhou)
    st = _lib.Status()
    f = fzeros(tuple(sim.intf.f.shape))
    f.copy_(sim.intf.f)
    sim.handle.call("ia_advect_momentum", ptr(f), ptr(u), ptr(u), ptr(old), C.c_double(0.25), C.c_int64(1), C.byref(st))
    return sim.intf.rhou[(slice(1, -1),) * D + (D - 1,)].clone()


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("arith", ["ff", "fp64"])
@pytest.mark.parametrize("limiter", LIMITERS)
@pytest.mark.parametrize("power", [-45, -60, -75])
def test_scaled_component(cuda, limiter, arith, power, D):
    one, small = advected(limiter, arith, 1.0, D), advected(limiter, arith, 2.0 ** power, D)
    assert bool(torch.isfinite(small).all())
    assert float((small * 2.0 ** -power - one).abs().max()) <= 1e-12 * float(one.abs().max())
