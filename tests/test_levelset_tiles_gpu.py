"""Redistancing on grids that leave remainders of the 32 x 8 blocks, against the oracle: noisy fields (every branch
of the upwind choice), fields that are flat away from a band (the gradient-free path), every kind of boundary, small
grids, and what the buffers hold afterwards.  1e-10 as in the other redistancing tests (FP64 sums of a few terms over
at most 24 stages).

Two cells between walls, or a ball centred in a periodic box, make second differences equal but for their rounding;
the minmod then goes one way or the other with it, in any implementation, so neither is compared here."""
import numpy as np
import pytest
import torch

import intfadv as ia
from intfadv import _lib
from intfadv.fields import ffrom, fzeros, ptr
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def npf(t):
    return np.asfortranarray(t.detach().cpu().numpy())


@pytest.mark.parametrize("dims,per", [((3, 4), ()), ((70, 19), (0,)), ((33, 9, 5), ()), ((65, 17, 6), (0, 1, 2)),
                                      ((31, 8, 40), (1,)), ((3, 3, 4), (2,))])
@pytest.mark.parametrize("kind", ["noise", "band"])
def test_redistance_matches_oracle(cuda, dims, per, kind):
    rng = np.random.default_rng(sum(dims))
    ng = tuple(n + 2 for n in dims)
    if kind == "noise":
        f = rng.random(ng)
    else:
        x = np.meshgrid(*[np.arange(n) - 0.5 for n in ng], indexing="ij")
        f = np.clip(0.5 - (np.sqrt(sum((xi - c * n) ** 2 for xi, n, c in zip(x, dims, (0.47, 0.53, 0.44)))) - 0.25 * min(dims)), 0, 1)
    f = np.asfortranarray(f)
    for e, n in enumerate(ng):                         # consistent ghosts, as every field of a run has them
        lo, hi = (n - 2, 1) if e in per else (1, n - 2)
        idx = lambda k: tuple(k if q == e else slice(None) for q in range(len(ng)))   # noqa: E731
        f[idx(0)], f[idx(n - 1)] = f[idx(lo)], f[idx(hi)]
    d, dtau = 2.0, 0.25
    h = ia.Handle(ia.make_config(dims, perdir=per))
    gf, phi, phi0, ini, L = ffrom(f), fzeros(ng), fzeros(ng), fzeros(ng), fzeros(ng)
    _lib.check(h.call("ia_levelset_init", ptr(gf), ptr(phi), ptr(ini)), "ia_levelset_init")
    _lib.check(h.call("ia_redistance", ptr(phi), ptr(phi0), ptr(ini), ptr(L), d, dtau), "ia_redistance")
    ref = O.redistance(f, d=d, dtau=dtau, per=per)
    assert np.abs(npf(phi) - ref).max() < 1e-10 * max(1.0, np.abs(ref).max())
    assert np.abs(npf(phi0) - O.redistance(f, d=d - dtau, dtau=dtau, per=per)).max() < 1e-10 * max(1.0, np.abs(ref).max())
    inner = tuple(slice(1, -1) for _ in dims)
    Lz = npf(L)
    Lz[inner] = 0
    assert not Lz.any()                                # the last right-hand side, nothing on its ghosts
    assert bool(torch.isfinite(L).all())
