"""
Measured points in no order: their bands are applied side by side and the values go
to the points' own places.
"""

import numpy as np
import pytest


def _shuffled(nq, seed=0):
    order = np.random.default_rng(seed).permutation(nq)
    q = np.geomspace(0.004, 0.3, nq)
    return q, q[order], order


@pytest.mark.parametrize("q, ordered", [([0.1], True), ([0.1, 0.1, 0.2], True),
                                        ([0.3, 0.2, 0.1], True), ([0.1, 0.3, 0.2], False)])
def test_band_order(q, ordered):
    from sasmodels_b200.resolution import _band_order
    order = _band_order(np.array(q))
    assert (order is None) == ordered
    if not ordered:
        assert np.all(np.diff(np.array(q)[order]) >= 0)


@pytest.mark.gpu
@pytest.mark.parametrize("nq, sets", [(3, 1), (200, 1), (200, 3), (33, 500), (700, 65), (1000, 1300)])
def test_shuffled_points_have_the_values_of_sorted_ones(cuda, nq, sets):
    """One curve, few and many (both kernels), bit for bit; the fallback that
    forms the weights in every call to its rounding."""
    import torch
    from sasmodels_b200 import resolution as R
    q, qs, order = _shuffled(nq)
    qc = np.geomspace(0.003, 0.4, 2000)
    st = torch.cuda.current_stream()
    a, b = R.Pinhole1D(q, 0.04*q, q_calc=qc), R.Pinhole1D(qs, 0.04*qs, q_calc=qc)
    th = torch.rand((sets, len(a.q_calc)), dtype=torch.float64, device="cuda") + 0.5
    if sets > 1:
        want, got = a.apply_sets(th, st), b.apply_sets(th, st)
    else:
        want, got = a.apply(th[0])[None], b.apply(th[0])[None]
    assert torch.equal(got, want[:, torch.as_tensor(order, device="cuda")])
    limit = R.MAX_WEIGHTS
    try:
        R.MAX_WEIGHTS = -1
        c = R.Pinhole1D(qs, 0.04*qs, q_calc=qc)
        formed = c.apply_sets(th, st) if sets > 1 else c.apply(th[0])[None]
    finally:
        R.MAX_WEIGHTS = limit
    torch.testing.assert_close(got, formed, rtol=1e-13, atol=0)
