"""The forms that a pressure solve of a small grid takes: one launch, or many while launch times are recorded.

On one level (2D, odd, a side above 96 cells) there is one form alone, whatever is recorded and however the smoother is
set, and the bits are the same.  On a hierarchy the two do the same iteration: after three Krylov steps the pressures
differ by rounding alone, some 50 operations a V-cycle and cell over up to six levels (2e-5 of the largest pressure in
FP32, 1e-13 in FP64), and a solve takes as many steps, but for one where a residual lies at the tolerance.
"""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr
from test_ragged_multigrid_gpu import apply, system

pytestmark = pytest.mark.gpu


def solve(dims, perdir, poisson, sys_, tol, itmx, timing=False, smoother=None):
    L, z, _ = sys_
    h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=0.05))
    if poisson == "mixed":
        ia.set_poisson_coef16(h, False)     # the one-launch form reads FP32 coefficients
    if smoother:
        ia.set_smoother(h, *smoother)
    if timing:
        _lib.check(h.call("ia_timing", 1, None, None, 0), "ia_timing")
    x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
    n0 = _lib.load().ia_launch_count()
    h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), tol, itmx, C.byref(it), C.byref(res))
    x = x[(slice(1, -1),) * len(dims)]
    return x - x.mean(), it.value, _lib.load().ia_launch_count() - n0


ONE_LEVEL = [((161, 97), ()), ((99, 8), ()), ((131, 98), (1,)), ((255, 255), ())]


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,perdir", ONE_LEVEL)
def test_one_level_whatever_is_set(cuda, dims, perdir, poisson):
    sys_ = system(dims, perdir, lrho=0.05)
    x, it, n = solve(dims, perdir, poisson, sys_, 1e-8, 3000)
    jt, m = solve(dims, perdir, poisson, sys_, 1e-3, 3000)[1:]
    assert jt < it and m == n      # one launch, however many iterations
    for kw in (dict(timing=True), dict(smoother=("halfsweep", 1.0)), dict(smoother=("blocked", 1.0))):
        y, jt, m = solve(dims, perdir, poisson, sys_, 1e-8, 3000, **kw)
        assert jt == it and m == n and torch.equal(x, y)


HIERARCHY = [
    ((160, 96), (), "mixed"), ((61, 87), (), "mixed"), ((254, 250), (1,), "mixed"), ((41, 35, 30), (), "mixed"),
    ((32, 64, 32), (0, 2), "mixed"), ((33, 36, 50), (1,), "mixed"), ((60, 50), (0,), "fp64"), ((61, 55), (), "fp64"),
    ((16, 15, 14), (), "fp64"), ((12, 18, 16), (0, 1, 2), "fp64"),
    # levels that halve evenly, whose launches have kernels of their own
    ((32, 34, 38), (), "mixed"), ((40, 32, 32), (0, 1, 2), "mixed"), ((64, 8, 72), (1,), "mixed"), ((72, 64, 8), (2,), "mixed"),
    ((4, 80, 112), (0,), "mixed"),
]
# odd periodic extents: cells of one colour touch across the wrap
ODD_WRAPS = [((25, 26, 23), (0, 2), "mixed"), ((33, 17), (0, 1), "mixed"), ((95, 64), (0,), "mixed"), ((33, 17), (0, 1), "fp64"),
             ((27, 21, 7), (0, 1, 2), "fp64"), ((10, 35, 11), (1,), "fp64")]


@pytest.mark.parametrize("dims,perdir,poisson", HIERARCHY + ODD_WRAPS)
def test_one_launch_and_many(cuda, dims, perdir, poisson):
    sys_ = system(dims, perdir, lrho=0.05)
    a, ita, n = solve(dims, perdir, poisson, sys_, 1e-30, 3)
    b, itb, m = solve(dims, perdir, poisson, sys_, 1e-30, 3, timing=True)
    assert ita == itb == 3 and n < m
    assert n == solve(dims, perdir, poisson, sys_, 1e-30, 6)[2]     # the one-launch form was taken
    assert float((a - b).abs().max()) <= (1e-4 if poisson == "mixed" else 1e-12) * float(b.abs().max())
    ita, itb = (solve(dims, perdir, poisson, sys_, 1e-10, 400, timing=t)[1] for t in (False, True))
    assert abs(ita - itb) <= 1


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,most", [((255, 255), 400), ((257, 257), 30), ((61, 87), 30), ((161, 97), 400), ((2001, 8), 400)])
def test_density_ratio_of_a_thousand_beside_the_limits(cuda, dims, most, poisson):
    # the largest odd square on one level, the smallest on a hierarchy, a grid on either side of 96 cells, a long one; on one
    # level these take up to 20000 iterations, and the hierarchy ends what three quarters of the allowed ones did not
    L, z, Li = system(dims, ())
    h = ia.Handle(ia.make_config(dims, poisson=poisson, lrho=1e-3))
    x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
    _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), 1e-10, max(most, 200), C.byref(it), C.byref(res)), "ia_poisson_solve")
    assert it.value <= most
    assert float((z[1:-1, 1:-1] - apply(Li, x[1:-1, 1:-1])).abs().max()) <= 2e-10


SIZES = [((66, 34, 38), ()), ((64, 48, 40), (0, 1, 2)), ((128, 8, 72), (1,)), ((72, 128, 8), (2,)), ((130, 66, 10), (0, 1))]


@pytest.mark.parametrize("nu,omega", [((2, 2), 1.15), ((1, 1), 1.15), ((1, 1), 1.0), ((1, 2), 1.0)])
@pytest.mark.parametrize("dims,perdir", SIZES)
def test_fp16_coefficients_that_are_exact(cuda, dims, perdir, nu, omega):
    # coefficients 1/4, 1/2, 1: their FP16 copies are exact, and the kernels that read those do the same arithmetic
    L, z, _ = system(dims, perdir)
    L.copy_(torch.where(L > 0, torch.exp2(-torch.floor(torch.log2(L.clamp_min(1.0)) / 4)), 0.0))
    got = []
    for on in (False, True):
        h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson="mixed", lrho=0.05))
        ia.set_poisson_coef16(h, on)
        ia.set_smoother(h, "halfsweep", omega)
        _lib.check(h.call("ia_poisson_mg_params", nu[0], nu[1], 16), "ia_poisson_mg_params")
        x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
        h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), 1e-30, 4, C.byref(it), C.byref(res))
        got.append((x, res.value))
    assert got[0][1] == got[1][1] and torch.equal(got[0][0], got[1][0])


@pytest.mark.parametrize("dims,perdir", [((20, 18, 16), (0, 2)), ((60, 50), ()), ((99, 8), ())])
def test_many_iterations_take_launches_of_two_thousand(cuda, dims, perdir):
    # a tolerance out of reach: all allowed iterations, and no launch that holds the device for all of them
    sys_ = system(dims, perdir, lrho=0.05)
    a, ita, n = solve(dims, perdir, "mixed", sys_, 1e-30, 100)
    b, itb, m = solve(dims, perdir, "mixed", sys_, 1e-30, 4100)
    assert ita == 100 and itb == 4100
    assert m == n + (2 if len(dims) == 3 or dims[0] % 2 == 0 else 1)   # one level: 3075 of them, then 1025 on the hierarchy
    assert float((a - b).abs().max()) <= 1e-9 * float(b.abs().max())
