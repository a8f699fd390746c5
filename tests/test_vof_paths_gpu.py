"""GPU parity of the VOF sweeps where their arithmetic or their route changes with the size of the input, against the CPU
oracle.  Fractions are in [0, 1], so that 1e-10 (absolute) leaves 5e5 roundings; c̄ is exact.
"""
import numpy as np
import pytest
import torch

import intfadv as ia
from intfadv.fields import fzeros
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-10


def npf(t):
    return np.asfortranarray(t.detach().cpu().numpy())


def against_oracle(intf, u1, u2, dt, steps, per=(), rel=1.0):
    fo = npf(intf.f)
    D = fo.ndim
    for s in range(1, steps + 1):
        st = ia.advect_vof_raw(intf, intf.f, u1, u2, dt, s)
        ost, cbar, rhouf, *_ = O.advect_vof(fo, npf(u1), npf(u2), dt, O.dir_order(s, D), lrho=1e-3, scheme="WH", per=per)
        assert (st.flags & 7) == ((1 if ost.nan else 0) | (2 if ost.over else 0) | (4 if ost.under else 0))
        assert np.isfinite(npf(intf.f)).all()
        assert np.abs(npf(intf.f) - fo).max() < TOL
        assert np.abs(npf(intf.rhouf) - rhouf).max() <= TOL * rel
        assert (npf(intf.cbar).astype(int) == cbar.astype(int)).all()


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("speed", [1e-200, 1e-300, 3e-310])
def test_quotients_near_the_ends_of_the_range(cuda, D, speed):
    """A layer normal to the flow: the donor's reduced normal is |u| dt times a unit vector, so that the reciprocals of
    its sum leave the range of FP64; a mass flux is below 2 |u| and compared relative to that."""
    n = 12
    intf = ia.cVOF((n,) * D, InterfaceSDF=lambda x: x[0] - 0.45 * n)
    u = fzeros(tuple(intf.Ng) + (D,), torch.float64, "cuda")
    u[..., 0] = speed
    against_oracle(intf, u, u, 1.0, 2, rel=1e5 * speed)


@pytest.mark.parametrize("n,per,centre", [((190, 94, 86), (), (0.5, 0.5, 0.5)), ((191, 95, 87), (0, 1, 2), (0.02, 0.98, 0.0)),
                                          ((254, 89, 65), (0, 2), (0.99, 0.5, 0.99)), ((97, 160, 95), (1,), (0.0, 0.0, 1.0))])
@pytest.mark.parametrize("cfl", [0.45, 0.9])
def test_tiles_of_one_fluid(cuda, n, per, centre, cfl):
    """From 1.5 million cells on the tiles of one fluid are done in one pass: sizes with whole, ragged and ghost-only last
    tiles, interfaces at and across the boundaries, and velocities below and above the bound of that pass."""
    r = 0.2 * min(n)
    intf = ia.cVOF(n, perdir=per, InterfaceSDF=lambda x: torch.sqrt(
        sum((x[d] - centre[d] * n[d] - 0.137 * (d + 1)) ** 2 for d in range(3))) - r)
    g = torch.Generator().manual_seed(len(per))
    u1, u2 = (fzeros(tuple(intf.Ng) + (3,), torch.float64, "cuda") for _ in range(2))
    x = torch.meshgrid(*[torch.arange(m, dtype=torch.float64) for m in intf.Ng], indexing="ij")
    for u in (u1, u2):
        for d in range(3):
            k, ph = torch.randint(1, 4, (3,), generator=g), torch.rand(3, generator=g)
            u[..., d] = (cfl * torch.stack([torch.sin(6.283185307179586 * (k[e] * x[e] / intf.Ng[e] + ph[e]))
                                            for e in range(3)]).prod(0)).to("cuda")
    against_oracle(intf, u1, u2, 1.0, 3, per)
