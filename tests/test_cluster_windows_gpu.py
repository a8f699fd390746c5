"""Two-dimensional pressure solves in one launch, whose blocks write their neighbours' copies of x directly: rows shared
between blocks, rows longer than a block's share, walls and wraps in either dimension, one level and a hierarchy.  The
solution has to satisfy the operator written out in plain FP64 torch and to come out the same twice."""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr
from test_ragged_multigrid_gpu import apply, system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poisson", ["fp64", "mixed"])
@pytest.mark.parametrize("dims,perdir,lrho", [
    ((160, 96), (), 1e-3), ((160, 96), (0,), 1e-3), ((62, 66), (0, 1), 1e-3), ((254, 250), (1,), 1e-3),
    ((4, 1000), (1,), 0.1), ((2000, 4), (0,), 0.1), ((99, 30), (), 0.1), ((30, 99), (0,), 0.1), ((131, 98), (1,), 0.1),
])
def test_solution_satisfies_the_operator(cuda, dims, perdir, lrho, poisson):
    L, z, Li = system(dims, perdir, lrho=lrho)
    tol, got = 1e-8, []
    for _ in range(2):
        h = ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=lrho))
        x, it, res = fzeros(z.shape), C.c_int32(), C.c_double()
        _lib.check(h.call("ia_poisson_solve", ptr(x), ptr(z), ptr(L), tol, 2000, C.byref(it), C.byref(res)), "ia_poisson_solve")
        got.append(x)
    r = z[1:-1, 1:-1] - apply(Li, x[1:-1, 1:-1])
    # the FP64 mode stops on the recurrence's residual, which drifts from the true one by rounding alone
    assert float(r.abs().max()) <= 2 * tol
    assert torch.equal(got[0], got[1])
