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


def test_adam_pack_matches_adam_and_pack(cuda):
    """One launch for every tensor, the bf16 copies and both weight images
    against the per-tensor Adam and the packing kernels, bit for bit."""
    import torch
    from sasmodels_b200.surrogate import HID, NIN
    rng = np.random.default_rng(7)
    (a, *_), (b, *_) = _gpu_net(np.random.default_rng(8)), _gpu_net(np.random.default_rng(8))
    g = torch.Generator(device="cuda").manual_seed(3)
    lib, st = b.lib, b.stream.cuda_stream
    for step in range(1, 3):
        splits = 3
        grads = [torch.randn(splits*p.numel() if k < 4 else p.numel(), device="cuda", generator=g)
                 for k, p in enumerate(a.params)]
        torch.cuda.synchronize()
        a.apply_gradients(grads, 1e-2, splits)
        for k, p in enumerate(b.params):
            nb = NIN if k == 0 else HID
            b._check(lib.sasb200_adam(
                p.numel(), splits if k < 4 else 1, grads[k].data_ptr(), p.data_ptr(),
                b.m[k].data_ptr(), b.v[k].data_ptr(), 1e-2, 0.9, 0.999, 1e-8, step,
                b.Wb[k].data_ptr() if k < 4 else None, b.WTb[k].data_ptr() if k < 4 else None,
                HID if k < 4 else 0, nb if k < 4 else 0, st), "adam")
        b._pack_kernels()
        a.stream.synchronize()
        b.stream.synchronize()
        for u, v in zip(a.params + a.m + a.v + a.Wb + a.WTb + [a.img, a.img_t],
                        b.params + b.m + b.v + b.Wb + b.WTb + [b.img, b.img_t]):
            assert torch.equal(u, v)


def test_captured_batch_gather(cuda):
    """The gather kernel and index_select (taken for strided data) give the
    same step; rows past the data set are refused through the error flag."""
    import torch
    from sasmodels_b200.surrogate import MLP
    n, B = 1000, 256
    wide = torch.rand((n, 32), device="cuda").to(torch.bfloat16)
    y = torch.randn(n, device="cuda")
    idx = torch.randperm(n, device="cuda")[:B]
    nets = []
    for x in (wide[:, :16], wide[:, :16].contiguous()):
        net = MLP(seed=6)
        lo = torch.zeros_like(x)
        torch.cuda.synchronize()
        net.train_step(x[:B].contiguous(), lo[:B].contiguous(), y[:B], B, 1e-3)
        graph = net.capture_training(x, lo, y, B, 1e-3, 100, 1)
        for _ in range(3):
            loss = graph.step(idx)
        net.stream.synchronize()
        assert net.errors() == 0
        nets.append((net, float(loss.item()), graph))
    assert nets[0][1] == nets[1][1]
    for u, v in zip(nets[0][0].params, nets[1][0].params):
        assert torch.equal(u, v)
    bad = idx.clone()
    bad[5] = n
    net, _, graph = nets[1]
    torch.cuda.synchronize()
    graph.step(bad)
    net.stream.synchronize()
    assert net.errors() == 5


def test_captured_step_follows_load_state(cuda):
    """Weights set from outside after the capture are the ones it trains."""
    import torch
    from sasmodels_b200.surrogate import MLP
    B = 128
    x = torch.rand((B, 16), device="cuda").to(torch.bfloat16)
    lo, y = torch.zeros_like(x), torch.randn(B, device="cuda")
    idx = torch.arange(B, device="cuda")
    a, b = MLP(seed=1), MLP(seed=2)
    torch.cuda.synchronize()
    out = []
    for net, late in ((a, True), (b, False)):
        if not late:
            net.load_state(a_state)
            torch.cuda.synchronize()
        graph = net.capture_training(x, lo, y, B, 1e-3, 100, 1)
        if late:
            a_state = MLP(seed=9).state()
            net.load_state(a_state)
            torch.cuda.synchronize()
        loss = graph.step(idx)
        net.stream.synchronize()
        out.append((float(loss.item()), [p.clone() for p in net.params]))
    assert out[0][0] == out[1][0]
    for u, v in zip(out[0][1], out[1][1]):
        assert torch.equal(u, v)


@pytest.mark.parametrize("n, blocks", [(128*3, 2), (128*4 - 5, 2), (128*5, 2), (128*9 + 1, 4),
                                       (128*149, 0), (128*297 + 1, 0), (128*1500, 5)])
def test_serve_pairs_is_serve(cuda, n, blocks):
    """Pairs of CTAs with two tiles in flight against one tile at a time, bit
    for bit: one and several double tiles per cluster, odd counts of tiles and
    of double tiles, an odd limit of blocks; rows beyond n are not written."""
    import torch
    from sasmodels_b200.surrogate import pad128
    rng = np.random.default_rng(n)
    net, *_ = _gpu_net(rng)
    x, xlo, _, _ = _inputs(rng, n, pad128(n))
    torch.cuda.synchronize()
    net.serve(x, xlo, n, blocks=blocks)
    net._infer_out.fill_(float("nan"))
    torch.cuda.synchronize()
    a = net.serve(x, xlo, n, blocks=blocks)
    net.stream.synchronize()
    a = a.clone()
    torch.cuda.synchronize()
    b = net.serve(x, xlo, n, blocks=pad128(n)//128)     # one tile per CTA
    net.stream.synchronize()
    assert net.errors() == 0
    assert torch.equal(a[:n], b[:n])
    assert torch.isnan(a[n:]).all()
