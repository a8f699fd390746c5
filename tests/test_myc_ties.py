"""The MYC normal where two of its candidates are equal but for rounding.

Along a plane interface normal to x the candidates of the y and of the z columns have the same leading component.  With
rounding in the fractions the two differ in the last digits; the normal must not depend on which one is larger, and a
flow that does not vary along z must stay so: its variation is the rounding and what the pressure solve leaves
(tolerance 1e-12), while a normal that goes either way moves f by 1e-2.
"""
import numpy as np
import pytest
import torch

import intfadv as ia
from oracle import pyoracle as O


def plane(axis, seed):
    """Fractions of a plane normal to an axis, with rounding (1e-14) in the mixed cells."""
    rng = np.random.default_rng(seed)
    f = np.zeros((9, 9, 9))
    f[:4] = 1.0
    f[4] = 0.76 + 1e-14 * rng.uniform(-1, 1, (9, 9))
    return np.asfortranarray(np.moveaxis(f, 0, axis))


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_oracle_normal_of_a_plane_with_rounding(axis):
    f = plane(axis, axis)
    for _ in range(20):
        idx = [int(v) for v in np.random.default_rng(_).integers(1, 8, 3)]
        idx[axis] = 4
        n = O.normal(f, tuple(idx), "MYC")
        assert np.abs(n - np.eye(3)[axis]).max() < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_normal_of_a_plane_with_rounding(cuda, axis):
    f = plane(axis, 10 + axis)
    intf = ia.cVOF((7, 7, 7), normalScheme="MYC")
    intf.f.copy_(torch.from_numpy(f))
    ia.reconstruct_interface(intf)
    n = intf.nhat[1:-1, 1:-1, 1:-1].movedim(axis, 0)[3]
    n = n / n.abs().sum(-1, keepdim=True)
    assert float((n - torch.eye(3, dtype=n.dtype, device=n.device)[axis]).abs().max()) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1002, 1008, 1015, 1026])
def test_a_dam_that_does_not_vary_along_z_stays_so(cuda, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    dims = (41, 35, 30)
    a, b = 41 * (0.25 + 0.05 * rng.uniform(-1, 1)), 35 * (0.5 + 0.05 * rng.uniform(-1, 1))
    amp = 0.2 * (1 + 0.2 * rng.uniform(-1, 1))
    kx, ky = np.pi / 41, np.pi / 35

    def u0(i, x):
        if i == 0:
            return amp * torch.sin(kx * x[0]) * torch.cos(ky * x[1])
        return -amp * kx / ky * torch.cos(kx * x[0]) * torch.sin(ky * x[1]) if i == 1 else 0.0 * x[0]
    sim = ia.TwoPhaseSimulation(dims, (0.0,) * 3, 30.0, U=1.0, u0=u0, λρ=1e-3, λμ=1 / 55, ν=0.03, g=(0.0, -1 / 30, 0.0),
                                InterfaceSDF=lambda x: torch.maximum(x[0] - a, x[1] - b) + 0.0 * sum(x), poisson="mixed",
                                poisson_tol=1e-12, poisson_itmx=400, normalScheme="MYC", λ="vanAlbada1")
    for _ in range(3):
        ia.sim_step(sim)
        f = sim.intf.f[1:-1, 1:-1, 1:-1]
        assert float((f - f[..., :1]).abs().max()) < 1e-11
