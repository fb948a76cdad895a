"""
The training step's kernels on tiled planes (csrc/mlp_train.cuh) against the
row-major kernels (bit for bit) and against float64 sums of the same planes.
"""

import numpy as np
import pytest

from test_mlp import _gpu_net, _inputs

pytestmark = pytest.mark.gpu


def _rows(planes, n_pad):
    """Tiled planes [4][tiles][32 groups][128 rows][8] as [4][n_pad][256]."""
    t = planes[:4*n_pad*256].view(4, n_pad//128, 32, 128, 8)
    return t.permute(0, 1, 3, 2, 4).reshape(4, n_pad, 256)


@pytest.mark.parametrize("n", [1, 128, 300, 3000, 128*160 + 5])
def test_training_step_kernels(cuda, n):
    """Fewer rows than a tile, ragged, fewer tiles than splits, and more tiles
    than SMs (several tiles per CTA)."""
    import torch
    from sasmodels_b200.surrogate import HID, NIN, pad128
    rng = np.random.default_rng(n)
    net, *_ = _gpu_net(rng)
    net.huber = 0.7
    n_pad = pad128(n)
    x, xlo, _, _ = _inputs(rng, n, n_pad)
    y = torch.as_tensor(rng.normal(0, 1, n_pad), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    loss, dW, db, dwo, dbo = net.gradients(x, xlo, y, n)
    net.stream.synchronize()
    assert net.errors() == 0
    z, h, dz = [_rows(t, n_pad).clone() for t in (net.z_save, net.h_save, net.dz_save)]
    # the row-major kernels
    bf = dict(dtype=torch.bfloat16, device="cuda")
    f32 = dict(dtype=torch.float32, device="cuda")
    zr, hr, dr = [torch.zeros(4*n_pad*HID, **bf) for _ in range(3)]
    out, dout, sq = [torch.zeros(n_pad, **f32) for _ in range(3)]
    lib, st = net.lib, net.stream.cuda_stream
    torch.cuda.synchronize()
    net._check(lib.sasb200_mlp_serve(n, n_pad, x.data_ptr(), xlo.data_ptr(), net.img.data_ptr(),
                                     net._ptrs(net.b), net.w_out.data_ptr(),
                                     net.b_out.data_ptr(), out.data_ptr(), zr.data_ptr(),
                                     hr.data_ptr(), net.err.data_ptr(), 0, st), "serve")
    net._check(lib.sasb200_loss_grad(n, n_pad, out.data_ptr(), y.data_ptr(), 0.7,
                                     dout.data_ptr(), sq.data_ptr(), st), "loss")
    net._check(lib.sasb200_mlp_backward_p(n, n_pad, net.img_t.data_ptr(), net.w_out.data_ptr(),
                                          dout.data_ptr(), zr.data_ptr(), dr.data_ptr(),
                                          net.err.data_ptr(), 0, st), "backward_p")
    net.stream.synchronize()
    assert torch.equal(net.out[:n], out[:n]) and torch.equal(net.dout[:n_pad], dout)
    for tiled, rows in ((z, zr), (h, hr), (dz, dr)):
        assert torch.equal(tiled, rows.view(4, n_pad, HID))
    # every gradient against float64 sums over the same planes; FP32 sums of
    # K terms stay within a few K ulp of the sum of their magnitudes
    d64, h64 = dz.double(), h.double()
    inputs = [x.double(), h64[0], h64[1], h64[2]]

    def close(got, want, scale):
        bound = 1e-5*scale + 1e-30
        assert ((got.double() - want).abs() <= bound).all()
    for l in range(4):
        nb = NIN if l == 0 else HID
        got = dW[l].view(net.splits, HID, nb).double().sum(0)
        close(got, d64[l].T @ inputs[l], d64[l].abs().T @ inputs[l].abs())
        close(db[l], d64[l].sum(0), d64[l].abs().sum(0))
    do = dout.double()
    close(dwo, h64[3].T @ do, h64[3].abs().T @ do.abs())
    close(dbo, do.sum().reshape(1), do.abs().sum())
    close(loss, sq[:n].double().mean(), sq[:n].double().mean())
    # the same gradients as one set of plain tensors
    red = net.reduced_gradients(x, xlo, y, n)
    net.stream.synchronize()
    assert torch.equal(red[0][0], loss) and torch.equal(red[10], dbo)
    for l in range(4):
        assert torch.equal(red[5 + l], db[l])
        close(red[1 + l], dW[l].view(net.splits, -1).double().sum(0),
              dW[l].view(net.splits, -1).double().abs().sum(0))
