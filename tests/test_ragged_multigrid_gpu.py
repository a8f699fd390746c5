"""The pressure multigrid on sizes that do not halve evenly.

Odd extents leave a single cell at the end of a coarse dimension, periodic extents coarsen to an even number
of cells, and an odd periodic extent of the grid itself puts cells of one colour beside each other across
the wrap.  On each the solve has to reach its tolerance in a number of iterations that belongs to a multigrid
(a single-level smoother needs 65 to 180 on grids of this size), to satisfy the operator written out in plain
FP64 torch, and to give the same bits twice.  Two-dimensional grids with an odd extent and a side above 96
cells are solved on one level, which takes many more iterations: the same checks at a droplet's density ratio.
"""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr

pytestmark = pytest.mark.gpu
TOL = 1e-10


def system(dims, perdir, seed=0, lrho=1e-3):
    """Face coefficients 1/ρ of two bubbles (zero on walls) and the divergence of random face values."""
    D = len(dims)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5).view([-1 if e == d else 1 for e in range(D)])
         for d, n in enumerate(dims)]
    dist = [torch.sqrt(sum((xi - n * c) ** 2 for xi, n in zip(x, dims))) for c in (0.3, 0.7)]
    f = torch.clamp(torch.minimum(*dist) - 0.2 * min(dims) + 0.5, 0, 1)
    rho = lrho + (1 - lrho) * f
    L, z = fzeros(tuple(n + 2 for n in dims) + (D,)), fzeros(tuple(n + 2 for n in dims))
    inner = (slice(1, -1),) * D
    Li = []
    for d in range(D):
        Ld = 2.0 / (rho + rho.roll(1, d))
        v = 0.01 * torch.randn(rho.shape, generator=gen, dtype=torch.float64, device="cuda")
        if d not in perdir:
            Ld.narrow(d, 0, 1).zero_()
            v.narrow(d, 0, 1).zero_()
        L[..., d][inner] = Ld
        hi = L[..., d].narrow(d, dims[d] + 1, 1)
        hi[tuple(slice(None) if e == d else slice(1, -1) for e in range(D))] = Ld.narrow(d, 0, 1)
        z[inner] += v.roll(-1, d) - v
        Li.append(Ld)
    return L, z, Li


def apply(Li, x):
    out = torch.zeros_like(x)
    for d, Ld in enumerate(Li):
        flux = Ld * (x.roll(1, d) - x)
        out += flux - flux.roll(-1, d)
    return out


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,perdir,most", [
    ((61, 87), (), 30),        # odd in both
    ((33, 17), (0, 1), 30),         # odd and periodic in both: colours meet across both wraps
    ((130, 50), (0,), 30),          # a periodic extent with an odd half
    ((41, 35, 30), (), 35),
    ((25, 50, 100), (0, 2), 35),    # odd periodic beside a wall and an even periodic extent
    ((27, 21, 19), (0, 1, 2), 35),  # odd and periodic in all three
    ((300, 2), (), 30),             # a dimension of two cells stays while the other halves
    ((40, 46, 24), (0, 2), 35),
])
def test_solve_converges_like_multigrid(cuda, dims, perdir, most, poisson):
    L, z, Li = system(dims, perdir)
    got = []
    for _ in range(2):
        h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=1e-3))
        x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
        _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), TOL, 400, C.byref(it), C.byref(res)),
                   "ia_poisson_solve")
        assert it.value <= most, it.value
        got.append(x)
    inner = (slice(1, -1),) * len(dims)
    r = z[inner] - apply(Li, x[inner])
    # the FP64 mode stops on the recurrence's residual, which drifts from the true one by rounding alone
    assert float(r.abs().max()) <= 2 * TOL
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,perdir", [((161, 97), ()), ((98, 45), (0,)), ((99, 8), ())])
def test_one_level_grids(cuda, dims, perdir, poisson):
    L, z, Li = system(dims, perdir, lrho=0.1)
    got, tol = [], 1e-8
    for _ in range(2):
        h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=0.1))
        x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
        _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), tol, 4000, C.byref(it), C.byref(res)),
                   "ia_poisson_solve")
        got.append(x)
    inner = (slice(1, -1),) * len(dims)
    assert float((z[inner] - apply(Li, x[inner])).abs().max()) <= 2 * tol
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("nu,omega", [((1, 1), 1.0), ((1, 0), 1.15), ((3, 2), 1.15)])
def test_smoothing_counts_on_odd_periodic_grids(cuda, nu, omega):
    dims, perdir = (25, 26, 23), (0, 2)
    L, z, Li = system(dims, perdir)
    h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson="mixed", lrho=1e-3))
    ia.set_smoother(h, "halfsweep", omega)
    _lib.check(h.call("ia_poisson_mg_params", nu[0], nu[1], 16), "ia_poisson_mg_params")
    x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
    _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), TOL, 400, C.byref(it), C.byref(res)),
               "ia_poisson_solve")
    assert float((z[1:-1, 1:-1, 1:-1] - apply(Li, x[1:-1, 1:-1, 1:-1])).abs().max()) <= 2 * TOL


@pytest.mark.parametrize("slab", [8, 16])
def test_slab_wavefront_on_a_grid_of_many_launches(cuda, slab):
    # the slabs apply where the half-sweeps are launches of their own (more than 65536 cells): the same bits
    dims, perdir = (64, 46, 40), (0, 2)
    L, z, _ = system(dims, perdir)
    got = []
    for rows in (0, slab):
        h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson="mixed", lrho=1e-3))
        ia.set_poisson_slab_rows(h, rows)
        x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
        _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), TOL, 400, C.byref(it), C.byref(res)),
                   "ia_poisson_solve")
        got.append((x, it.value, res.value))
    assert got[0][1:] == got[1][1:] and torch.equal(got[0][0], got[1][0])
