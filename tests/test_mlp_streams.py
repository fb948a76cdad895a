"""
Weights set from outside are in order with the network's own stream, without
a synchronisation by the caller.
"""

import numpy as np
import pytest

from test_mlp import _inputs

pytestmark = pytest.mark.gpu
CYCLES = 40_000_000          # some 20 ms of a stream's time


def _state(net):
    return {k: [t.clone() for t in v] if isinstance(v, list) else v.clone()
            for k, v in (("W", net.W), ("b", net.b), ("w_out", net.w_out), ("b_out", net.b_out))}


def test_serve_after_load_state(cuda):
    """The weights come late on the caller's stream: serve waits for them."""
    import torch
    from sasmodels_b200.surrogate import MLP
    x, xlo, _, _ = _inputs(np.random.default_rng(0), 1000, 1024)
    want_net, net = MLP(seed=5), MLP(seed=6)
    state = _state(want_net)
    torch.cuda.synchronize()
    want = want_net.serve(x, xlo, 1000)[:1000]
    net.serve(x, xlo, 1000)
    torch.cuda.synchronize()
    late = {k: [torch.zeros_like(t) for t in v] if isinstance(v, list) else torch.zeros_like(v)
            for k, v in state.items()}
    torch.cuda.synchronize()
    torch.cuda._sleep(CYCLES)
    for k, v in state.items():
        for a, b in zip(late[k], v) if isinstance(v, list) else [(late[k], v)]:
            a.copy_(b)
    net.load_state(late)
    got = net.serve(x, xlo, 1000)[:1000]
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("batch", [128, 128*80])
def test_load_state_between_steps(cuda, batch):
    """A captured step is still queued on the network's stream when the weights
    are set; the next step trains the new ones."""
    import torch
    from sasmodels_b200.surrogate import MLP
    x = torch.rand((batch, 16), device="cuda").to(torch.bfloat16)
    lo, y = torch.zeros_like(x), torch.randn(batch, device="cuda")
    idx = torch.arange(batch, device="cuda")
    results = []
    for wait in (True, False):
        net, other = MLP(seed=1), MLP(seed=9)
        torch.cuda.synchronize()
        graph = net.capture_training(x, lo, y, batch, 1e-3, 100, 1)
        torch.cuda.synchronize()
        with torch.cuda.stream(net.stream):
            torch.cuda._sleep(CYCLES)
        graph.step(idx)
        if wait:
            torch.cuda.synchronize()
        net.load_state(_state(other))
        if wait:
            torch.cuda.synchronize()
        loss = graph.step(idx)
        torch.cuda.synchronize()
        assert net.errors() == 0
        results.append([loss.clone()] + [t.clone() for t in net.params + net.m + net.v + net.Wb
                                         + [net.img, net.img_t]])
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("batch", [128, 128*80])
def test_loss_of_a_captured_step_on_the_callers_stream(cuda, batch):
    """The loss is read while the step is still to come on the network's stream."""
    import torch
    from sasmodels_b200.surrogate import MLP
    x = torch.rand((batch, 16), device="cuda").to(torch.bfloat16)
    lo, y = torch.zeros_like(x), torch.randn(batch, device="cuda")
    idx = torch.arange(batch, device="cuda")
    net = MLP(seed=1)
    torch.cuda.synchronize()
    graph = net.capture_training(x, lo, y, batch, 1e-3, 100, 1)
    torch.cuda.synchronize()
    for _ in range(2):
        with torch.cuda.stream(net.stream):
            torch.cuda._sleep(CYCLES)
        got = float(graph.step(idx).item())
        torch.cuda.synchronize()
        assert got == float(graph.loss.item()) and got > 0
