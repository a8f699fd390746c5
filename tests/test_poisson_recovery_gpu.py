"""A handle after a solve that ended in NaN: the next solves, in either form, are as on a new handle."""
import ctypes as C

import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import fzeros, ptr
from test_ragged_multigrid_gpu import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("dims,perdir,poisson", [((16, 18, 20), (0, 2), "mixed"), ((33, 24, 10), (0, 1, 2), "mixed"),
                                                 ((12, 14, 16), (0, 2), "fp64"), ((60, 50), (0,), "fp64"),
                                                 ((60, 50), (0, 1), "mixed"), ((13, 14, 11), (0,), "fp64")])
def test_solve_after_a_solve_that_diverged(cuda, dims, perdir, poisson, timing, bad):
    L, z, _ = system(dims, perdir, lrho=0.05)
    z_bad = fzeros(z.shape)
    z_bad.copy_(z)
    z_bad[(3,) * len(dims)] = bad
    x = fzeros(z.shape)

    def solve(h, rhs):
        it, res = C.c_int32(), C.c_double()
        x.zero_()
        code = h.call("ia_poisson_solve", ptr(x), ptr(rhs), ptr(L), 1e-9, 60, C.byref(it), C.byref(res))
        return code, it.value, res.value, x.clone()
    fresh, used = (ia.Handle(ia.make_config(dims, perdir=perdir, poisson=poisson, lrho=0.05)) for _ in range(2))
    assert solve(used, z_bad)[0] == _lib.IA_WARN_NOT_CONVERGED
    for h in (fresh, used):
        _lib.check(h.call("ia_timing", int(timing), None, None, 0), "ia_timing")
    a, b = solve(fresh, z), solve(used, z)
    assert a[0] == b[0] == 0 and a[1:3] == b[1:3] and torch.equal(a[3], b[3])
