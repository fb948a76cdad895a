"""
Rounding of the weight gradients' sums over the rows: short accumulation chains
on the tensor core, whatever the size of the batch.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 2048, 2049, 4097, 6144, 6145, 8192, 65536])
def test_gradients_against_float64_sums(cuda, n):
    """Against float64 sums over the same planes, at the edges of the rule for the
    chains.  A chain of at most 256 rows adds 16 times, each time losing less than
    an ulp (2^-23) of a sum that grows to its value: 1e-6 of it at most on
    average; a whole split of 65,536 rows in one chain would lose 25 times that.
    Sums in FP32 and double precision stay within a few roundings."""
    import torch
    from sasmodels_b200.surrogate import HID, MLP, pad128
    g = torch.Generator(device="cuda").manual_seed(n)
    n_pad = pad128(n)
    xf = torch.rand((n_pad, 16), device="cuda", generator=g)*2 - 1
    xf[n:] = 0
    x = xf.bfloat16()
    x_lo = (xf - x.float()).bfloat16()
    y = 0.3*torch.randn(n_pad, device="cuda", generator=g)
    net = MLP(seed=1)
    net.huber = 0.02
    torch.cuda.synchronize()
    red = net.reduced_gradients(x, x_lo, y, n)
    torch.cuda.synchronize()
    assert net.errors() == 0

    def plane(t, l):
        t = t[:4*n_pad*HID].view(4, n_pad//128, 32, 128, 8)[l]
        return t.permute(0, 2, 1, 3).reshape(n_pad, HID).double()

    def off(got, want):
        return float((got.double().view_as(want) - want).norm()/want.norm())
    dout = net.dout[:n_pad].double()
    for l in range(4):
        d = plane(net.dz_save, l)
        h = x.double() if l == 0 else plane(net.h_save, l - 1)
        assert off(red[1 + l], d.T @ h) < 1e-6
        assert off(red[5 + l], d.sum(0)) < 2e-7
    assert off(red[9], plane(net.h_save, 3).T @ dout) < 2e-7
    assert abs(float(red[10].double() - dout.sum())) < 4e-7*float(dout.abs().sum())
    d = (net.out[:n].double() - y[:n].double()).abs()
    loss = float(torch.where(d <= 0.02, d*d, 0.02*(2*d - 0.02)).mean())
    assert abs(float(red[0]) - loss) < 4e-7*loss
