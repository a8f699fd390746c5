"""The order of the FP32 forward pass: every output is one chain of multiply-adds from the bias, tap by tap with the
channels inside.  A unit whose input is zero but for rounding is on or off by that order, and with it a part of the
gradient, so the order is part of the result: the network's output has to come out bit for bit.
"""
import pytest
import torch

from intfadv import learned
from test_learned_train_gpu import case, weights

pytestmark = pytest.mark.gpu


def fma32(w, x, acc):
    """fma(w, x, acc) on FP32 values: the product is exact in FP64; the sum is rounded to odd there and then to FP32."""
    p, a = w.double() * x.double(), acc.double()
    s = p + a
    t = s - p
    e = (p - (s - t)) + (a - t)
    bits = s.view(torch.int64)
    cut = bits - ((e * s.sign()) < 0).to(torch.int64)
    return torch.where(e != 0, (cut | 1).view(torch.float64), s).float()


def chain(params, l, v):
    """Layer l on v[B, z, y, x, c], zero padding."""
    ci, co = learned.CIN[l], learned.COUT[l]
    W, b = params[l]
    n = v.shape[1:4]
    v = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
    acc = b.expand(v.shape[0], *n, co).clone()
    for t in range(27):
        dz, dy, dx = t // 9, t // 3 % 3, t % 3
        part = v[:, dz:dz + n[0], dy:dy + n[1], dx:dx + n[2]]
        for c in range(ci):
            acc = fma32(W[t, :, c].expand_as(acc), part[..., c:c + 1].expand_as(acc), acc)
    return acc


def pool(v):
    s = torch.zeros_like(v[:, ::2, ::2, ::2])
    for k in range(8):
        s = s + v[:, k >> 2::2, (k >> 1) & 1::2, k & 1::2]
    return s * 0.125


def up(v):
    for e in (1, 2, 3):
        v = v.repeat_interleave(2, e)
    return v


@pytest.mark.parametrize("B,nx,ny,nz", [(1, 4, 4, 4), (1, 20, 12, 8), (2, 36, 20, 12), (1, 40, 24, 20)])
def test_forward_is_a_chain_in_the_order_of_the_taps(cuda, B, nx, ny, nz):
    x0, _ = case(B, nx, ny, nz)
    w = weights(1.0, 0.0, nx + ny + nz)
    net = learned.Net()
    net.set_params(w)
    wt, params = torch.tensor(w, dtype=torch.float32, device="cuda"), []
    for (wo, bo), ci, co in zip(learned.layer_offsets(), learned.CIN, learned.COUT):
        params.append((wt[wo:bo].view(27, co, ci), wt[bo:bo + co]))
    a1 = chain(params, 0, x0[:, 1:-1, 1:-1, 1:-1].contiguous()).relu()
    a2 = chain(params, 1, pool(a1)).relu()
    a3 = chain(params, 2, pool(a2)).relu()
    a4 = chain(params, 3, up(a3) + a2).relu()
    a5 = chain(params, 4, up(a4)).relu() + a1
    out = chain(params, 5, a5)[..., 0]
    assert torch.equal(net.forward(x0)[:, 1:-1, 1:-1, 1:-1], out)
