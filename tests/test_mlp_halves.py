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
