"""
Hand-overs between the two CTAs of a pair (csrc/mlp_pairs.cuh,
csrc/mlp_halves.cuh): every arrival on the other CTA's barrier releases, and
repeated runs give the values of one tile per CTA.
"""

import os
import re

import numpy as np
import pytest

from test_mlp import _gpu_net, _inputs

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sasmodels_b200", "csrc")


def _statements(name):
    """The asm statements of a source file, their strings joined."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return ["".join(re.findall(r'"([^"]*)"', s))
            for s in re.findall(r"asm volatile\((.*?)\);", text, re.S)]


@pytest.mark.parametrize("name", ["tc_ptx.cuh", "mlp_pairs.cuh", "mlp_halves.cuh", "mlp.cu"])
def test_remote_arrivals_release(name):
    """An arrival in another CTA releases at cluster scope, by itself or by a
    fence ahead of it in the same statement."""
    for s in _statements(name):
        at = s.find("mbarrier.arrive")
        if at >= 0 and "shared::cluster" in s[at:] and "tcgen05" not in s:
            assert "mbarrier.arrive.release.cluster" in s or re.search(
                r"fence\.(release|acq_rel)\S*\.cluster;.*mbarrier\.arrive\.relaxed\.cluster", s), s


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1000, 128*74, 128*149 + 3, 50021])
def test_serving_is_the_same_every_time(cuda, n):
    """Two SMs per tile up to 74 tiles, pairs with two tiles in flight beyond
    148: 200 runs, each in the place of other values."""
    import torch
    from sasmodels_b200.surrogate import pad128
    rng = np.random.default_rng(n)
    net, *_ = _gpu_net(rng)
    x, xlo, _, _ = _inputs(rng, n, pad128(n))
    torch.cuda.synchronize()
    # one tile per CTA, 128 tiles at a time
    want = torch.empty(n, device="cuda")
    for a in range(0, n, 128*128):
        b = min(n, a + 128*128)
        out = net.serve(x[a:pad128(b)], xlo[a:pad128(b)], b - a, blocks=(b - a + 127)//128)
        net.stream.synchronize()
        want[a:b] = out[:b - a]
        torch.cuda.synchronize()
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(net.stream):
        for k in range(200):
            net._infer_out.fill_(float(k))
            wrong += (net.serve(x, xlo, n)[:n] != want).sum()
    net.stream.synchronize()
    assert net.errors() == 0 and int(wrong) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3001, 128*74])
def test_gradients_are_the_same_every_time(cuda, n):
    """Forward and backward on two SMs per tile: 100 passes over planes that
    were overwritten in between."""
    import torch
    from sasmodels_b200.surrogate import pad128
    rng = np.random.default_rng(n)
    net, *_ = _gpu_net(rng)
    net.huber = 0.7
    x, xlo, _, _ = _inputs(rng, n, pad128(n))
    y = torch.as_tensor(rng.normal(0, 1, pad128(n)), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    want = None
    with torch.cuda.stream(net.stream):
        for k in range(100):
            got = net.reduced_gradients(x, xlo, y, n)
            if want is None:
                want = got
            for a, b in zip(got, want):
                wrong += (a != b).sum()
            for plane in (net.z_save, net.h_save, net.dz_save):
                plane.fill_(float(k))
    net.stream.synchronize()
    assert net.errors() == 0 and int(wrong) == 0
