"""
Few tiles on two SMs each (csrc/mlp_halves.cuh) against the kernels of one tile
per SM: the same values, on both sides of the rule that chooses.
"""

import numpy as np
import pytest

import test_mlp_train as train
from test_mlp import _gpu_net, _inputs

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("rows", ["1", "32", "64", "65", "128", "129", "1000",
                                  "all", "all - 63", "all + 1"])
def test_serve(cuda, rows):
    """`all`: the rows of as many tiles as are served by two SMs each at once."""
    import torch
    from sasmodels_b200.surrogate import pad128
    n = eval(rows, dict(all=_sms()//2*128))
    rng = np.random.default_rng(n)
    net, *_ = _gpu_net(rng)
    n_pad = pad128(n)
    x, xlo, _, _ = _inputs(rng, n, n_pad)
    out = [torch.full((n_pad,), -7.0, dtype=torch.float32, device="cuda") for _ in range(2)]
    net._pack()
    torch.cuda.synchronize()
    # 0: all SMs; a CTA per tile is too few for two per tile
    for o, blocks in zip(out, (0, n_pad//128)):
        net._check(net.lib.sasb200_mlp_serve(n, n_pad, x.data_ptr(), xlo.data_ptr(),
                                             net.img.data_ptr(), net._ptrs(net.b),
                                             net.w_out.data_ptr(), net.b_out.data_ptr(),
                                             o.data_ptr(), None, None, net.err.data_ptr(), blocks,
                                             net.stream.cuda_stream), "serve")
    net.stream.synchronize()
    assert net.errors() == 0
    assert torch.equal(*out) and (out[0][n:] == -7.0).all() and (out[0][:n] != -7.0).all()


@pytest.mark.parametrize("extra", [-63, 1])
def test_training_step(cuda, extra):
    """The last batch that has two SMs per tile, and the first that has not."""
    train.test_training_step_kernels(cuda, _sms()//2*128 + extra)


@pytest.mark.parametrize("tiles", [1, 0, "more"])
def test_captured_batch(cuda, tiles):
    """The forward that gathers its batch (tiles 0: the most it takes) and, from one
    tile more on, the gathering launch, against index_select (strided data)."""
    import torch
    from sasmodels_b200.surrogate import MLP
    B = 128*(_sms()//2 + 1 if tiles == "more" else tiles or _sms()//2)
    n = B + 77
    wide = torch.rand((n, 32), device="cuda").to(torch.bfloat16)
    y = torch.randn(n, device="cuda")
    idx = torch.randint(0, n, (B,), device="cuda")
    done = []
    for x in (wide[:, :16], wide[:, :16].contiguous()):
        net = MLP(seed=4)
        lo = torch.full_like(x, 2.0**-9)
        torch.cuda.synchronize()
        graph = net.capture_training(x, lo, y, B, 1e-3, 100, 1)
        losses = [float(graph.step(idx).item()) for _ in range(2)]
        net.stream.synchronize()
        assert net.errors() == 0
        done.append((net, losses, graph))
    assert done[0][1] == done[1][1]
    for u, v in zip(done[0][0].params, done[1][0].params):
        assert torch.equal(u, v)
    for name in ("xb", "xlb", "yb", "counters", "sched"):
        assert torch.equal(getattr(done[0][2], name), getattr(done[1][2], name))
    net, _, graph = done[1]
    idx[B - 1] = -1
    torch.cuda.synchronize()
    graph.step(idx)
    net.stream.synchronize()
    assert net.errors() == 5
    assert (graph.xb[B - 1] == 0).all() and graph.yb[B - 1] == 0
