"""
A captured training step whose batch names a row outside the data set trains
nothing and says so, in the step itself and in those that follow; features
padded to whole tiles are gathered like others.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [128, 128*80])
@pytest.mark.parametrize("row", [-1, 1000, 1 << 40])
@pytest.mark.parametrize("huber", [0.0, 0.5])
def test_row_outside_trains_nothing(cuda, batch, row, huber):
    """The forward that gathers its batch (128 rows) and the gathering kernel;
    just outside on either side and far outside."""
    import torch
    from sasmodels_b200.surrogate import MLP
    n = 1000
    x = torch.rand((n, 16), device="cuda").to(torch.bfloat16)
    lo, y = torch.zeros_like(x), torch.randn(n, device="cuda")
    idx = torch.randint(0, n, (batch,), device="cuda")
    bad = idx.clone()
    bad[batch - 3] = row
    net = MLP(seed=3)
    net.huber = huber
    torch.cuda.synchronize()
    graph = net.capture_training(x, lo, y, batch, 1e-3, 100, 1)
    first = graph.step(idx)
    torch.cuda.synchronize()
    assert torch.isfinite(first)
    kept = [t.clone() for t in net.params + net.m + net.v + net.Wb + net.WTb
            + [net.img, net.img_t]]
    torch.cuda.synchronize()
    with torch.cuda.stream(net.stream):
        torch.cuda._sleep(200_000_000)
    graph.step(bad)
    loss = graph.step(idx)           # queued before the host can know
    torch.cuda.synchronize()
    assert torch.isnan(loss) and net.errors() == 5
    with pytest.raises(RuntimeError, match="outside the training data"):
        graph.step(idx)
    torch.cuda.synchronize()
    for a, b in zip(kept, net.params + net.m + net.v + net.Wb + net.WTb + [net.img, net.img_t]):
        assert torch.equal(a, b)
    # the network goes on with another graph
    again = net.capture_training(x, lo, y, batch, 1e-3, 100, 1)
    loss = again.step(idx)
    torch.cuda.synchronize()
    assert torch.isfinite(loss) and net.errors() == 0
    assert not torch.equal(kept[0], net.params[0])


@pytest.mark.parametrize("batch", [128, 128*80])
@pytest.mark.parametrize("n", [1, 1000, 1024])
def test_padded_features_are_gathered(cuda, batch, n):
    """n targets with the padded features of MLP.features, as the surrogate trains,
    against index_select (strided data); the padding is outside the data set."""
    import torch
    from sasmodels_b200.surrogate import MLP, pad128
    wide = torch.rand((pad128(n), 32), device="cuda").to(torch.bfloat16)
    y = torch.randn(n, device="cuda")
    idx = torch.randint(0, n, (batch,), device="cuda")
    results = []
    for x in (wide[:, :16].contiguous(), wide[:n, :16]):
        net = MLP(seed=4)
        lo = torch.full_like(x, 2.0**-9)
        torch.cuda.synchronize()
        graph = net.capture_training(x, lo, y, batch, 1e-3, 100, 1)
        assert graph.direct == x.is_contiguous()
        for _ in range(2):
            loss = graph.step(idx)
        torch.cuda.synchronize()
        assert net.errors() == 0
        results.append([loss.clone()] + [t.clone() for t in net.params + net.m + net.v])
        if graph.direct and n < len(x):
            idx_pad = idx.clone()
            idx_pad[0] = n
            torch.cuda.synchronize()
            loss = graph.step(idx_pad)
            torch.cuda.synchronize()
            assert torch.isnan(loss) and net.errors() == 5
    for a, b in zip(*results):
        assert torch.equal(a, b)
