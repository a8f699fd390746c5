"""The FP32 training kernels at the edges of their tiles, against the network in plain FP64 torch.

The convolutions tile 32 x 8 x 4 cells (2 planes on small grids, 16 cells along x on short rows), the weight
gradient 16 x 4 x 2; the sizes below leave remainders of each along every dimension and take every tile.
Tolerances as in the oracle tests of the same kernels: 2e-6 of the largest output, 5e-5 of the largest gradient
of a layer (FP32 sums over up to 864 products and, for a gradient, over all cells).

The gradients are taken where every ReLU is active: a unit whose input is within FP32 rounding of zero is on or
off by chance, and one such unit in a grid of 10^4 cells moves a gradient by 1e-4 whatever the kernels do.
"""
import numpy as np
import pytest
import torch

from intfadv import learned

pytestmark = pytest.mark.gpu


def reference(w, x0, tgt):
    params, lowest, o = [], [], 0
    for ci, co in zip(learned.CIN, learned.COUT):
        n = 27 * co * ci
        params.append(torch.tensor(w[o:o + n], dtype=torch.float64, device="cuda").view(27, co, ci).requires_grad_())
        params.append(torch.tensor(w[o + n:o + n + co], dtype=torch.float64, device="cuda").requires_grad_())
        o += n + co

    def conv(v, l):
        n = v.shape[1:4]
        v = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        out = params[2 * l + 1]
        for t in range(27):
            dz, dy, dx = t // 9, t // 3 % 3, t % 3
            out = out + v[:, dz:dz + n[0], dy:dy + n[1], dx:dx + n[2]] @ params[2 * l][t].T
        lowest.append(float(out.detach().min()))
        return out

    def pool(v):
        B, nz, ny, nx, c = v.shape
        return v.view(B, nz // 2, 2, ny // 2, 2, nx // 2, 2, c).mean((2, 4, 6))

    def up(v):
        for e in (1, 2, 3):
            v = v.repeat_interleave(2, e)
        return v
    x = x0[:, 1:-1, 1:-1, 1:-1].double()
    a1 = conv(x, 0).relu()
    a2 = conv(pool(a1), 1).relu()
    a4 = conv(up(conv(pool(a2), 2).relu()) + a2, 3).relu()
    out = conv(conv(up(a4), 4).relu() + a1, 5)[..., 0]
    loss = ((out - tgt[:, 1:-1, 1:-1, 1:-1].double()) ** 2).mean()
    loss.backward()
    return out.detach(), float(loss.detach()), [p.grad.reshape(-1) for p in params], min(lowest[:5])


SIZES = [
    (1, 4, 4, 4),         # the smallest
    (1, 20, 12, 8),       # 2-plane tiles, short rows below
    (2, 36, 20, 12),      # remainders along x, y and z
    (1, 68, 28, 20),
    (2, 52, 76, 84),      # 4-plane tiles at full resolution
]


def case(B, nx, ny, nz):
    gen = torch.Generator(device="cuda").manual_seed(nx)
    x0 = torch.zeros((B, nz + 2, ny + 2, nx + 2, 4), device="cuda")
    x0[:, 1:-1, 1:-1, 1:-1] = torch.randn((B, nz, ny, nx, 4), generator=gen, device="cuda")
    tgt = torch.zeros(x0.shape[:-1], device="cuda")
    tgt[:, 1:-1, 1:-1, 1:-1] = torch.randn((B, nz, ny, nx), generator=gen, device="cuda")
    return x0, tgt


def weights(scale, bias, seed):
    rng = np.random.default_rng(seed)
    w = learned.init_params(5)
    for (wo, bo), co in zip(learned.layer_offsets(), learned.COUT):
        w[wo:bo] *= scale
        w[bo:bo + co] = bias + 0.1 * rng.standard_normal(co)
    return w


@pytest.mark.parametrize("B,nx,ny,nz", SIZES)
def test_forward_at_tile_edges(cuda, B, nx, ny, nz):
    x0, tgt = case(B, nx, ny, nz)
    w = weights(1.0, 0.0, nx + ny + nz)
    net = learned.Net()
    net.set_params(w)
    ref, loss, _, _ = reference(w, x0, tgt)
    out = net.forward(x0)
    assert float((out[:, 1:-1, 1:-1, 1:-1] - ref).abs().max() / ref.abs().max()) < 2e-6
    out[:, 1:-1, 1:-1, 1:-1] = 0
    assert not bool(out.any())     # the halo stays zero
    got, g = net.loss_grad(x0, tgt)
    assert abs(got - loss) < 1e-5 * loss
    assert torch.equal(g, net.loss_grad(x0, tgt)[1])      # sums in a fixed order


@pytest.mark.parametrize("B,nx,ny,nz", SIZES)
def test_gradients_at_tile_edges(cuda, B, nx, ny, nz):
    x0, tgt = case(B, nx, ny, nz)
    w = weights(0.1, 5.0, nx + ny + nz)
    net = learned.Net()
    net.set_params(w)
    _, loss, grads, lowest = reference(w, x0, tgt)
    assert lowest > 0.01           # every unit is on
    got, g = net.loss_grad(x0, tgt)
    assert abs(got - loss) < 1e-5 * loss
    o = 0
    for l, r in enumerate(grads):
        e = float((g[o:o + r.numel()] - r).abs().max() / r.abs().max())
        assert e < 5e-5, (l, e)
        o += r.numel()
