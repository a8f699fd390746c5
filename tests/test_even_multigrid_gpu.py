"""The FP32 smoother, restriction and matrix product of levels that halve evenly, against independent kernels.

At relaxation 1 the half-sweeps do the temporally blocked smoother's arithmetic, which has its own kernel and the
general restriction.  After three Krylov steps the two pressures differ by FP32 rounding alone: some 50 operations a
V-cycle and cell, over six levels, at 6e-8 each are 2e-5, and a wrong neighbour, wrap or coefficient moves the pressure
by percents.  With over-relaxation (the default) the solve has to reach its tolerance in a multigrid's number of steps.
"""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr
from test_ragged_multigrid_gpu import apply, system

pytestmark = pytest.mark.gpu
SIZES = [((66, 34, 38), ()), ((64, 48, 40), (0, 1, 2)), ((128, 8, 72), (1,)), ((8, 128, 72), (0,)), ((72, 128, 8), (2,)),
         ((4, 160, 112), (0, 2)), ((130, 66, 10), (0, 1))]


def solve(dims, perdir, L, z, smoother, omega, coef16, tol, itmx):
    h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson="mixed", lrho=1e-3))
    ia.set_poisson_coef16(h, coef16)
    ia.set_smoother(h, smoother, omega)
    x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
    code = h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), tol, itmx, C.byref(it), C.byref(res))
    return x[1:-1, 1:-1, 1:-1], it.value, code


@pytest.mark.parametrize("dims,perdir", SIZES)
def test_half_sweeps_match_the_blocked_smoother(cuda, dims, perdir):
    L, z, _ = system(dims, perdir, lrho=0.05)
    a, ita, _ = solve(dims, perdir, L, z, "halfsweep", 1.0, False, 1e-30, 3)
    b, itb, _ = solve(dims, perdir, L, z, "blocked", 1.0, False, 1e-30, 3)
    assert ita == itb == 3
    a, b = a - a.mean(), b - b.mean()
    assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max())


@pytest.mark.parametrize("coef16", [False, True])
@pytest.mark.parametrize("dims,perdir", SIZES)
def test_relaxed_half_sweeps_converge(cuda, dims, perdir, coef16):
    L, z, Li = system(dims, perdir)
    x, it, code = solve(dims, perdir, L, z, "halfsweep", 1.15, coef16, 1e-10, 400)
    _lib.check(code, "ia_poisson_solve")
    assert it <= 35
    assert float((z[1:-1, 1:-1, 1:-1] - apply(Li, x)).abs().max()) <= 1e-10 * 1.01
