"""Pressure solves whose right-hand side has a mean, which no pressure can balance: the residual that a solve returns is
that of the pressure it returns, and the code says that the tolerance is not met.  On one level (2D, odd, a side above
96 cells) and on a hierarchy, in one launch and in many."""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr
from test_ragged_multigrid_gpu import apply, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,perdir", [((99, 8), ()), ((8, 99), (0,)), ((161, 97), ()), ((61, 87), ()), ((64, 48), (0,)),
                                         ((20, 18, 11), ()), ((160, 144), ())])
@pytest.mark.parametrize("mean", [1e-3, 0.0])
def test_residual_of_the_returned_pressure(cuda, dims, perdir, poisson, mean):
    L, z, Li = system(dims, perdir, lrho=0.1)
    inner = (slice(1, -1),) * len(dims)
    z[inner] += mean - z[inner].mean()
    h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=0.1))
    x, it, res, tol, most = fzeros(z.shape), C.c_int32(), C.c_double(), 1e-8, 60 if mean else 2000
    code = h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), tol, most, C.byref(it), C.byref(res))
    true = float((z[inner] - apply(Li, x[inner])).abs().max())
    # the FP64 mode's residual is the recurrence's: rounding of x and of the products, each iteration
    size = float((max(float(l.abs().max()) for l in Li) * x[inner].abs()).max()) + float(z.abs().max())
    assert abs(res.value - true) <= 1e-14 * it.value * size + 1e-15
    assert (code == _lib.IA_WARN_NOT_CONVERGED) == bool(mean)
    assert not mean or true >= 0.99 * mean
