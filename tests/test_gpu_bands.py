"""
The banded-weight plans of the resolution classes (csrc/resolution.cu:
pinhole_weights, slit_weights, band_apply, band_apply_sets) and the
many-curve nllf against the dense-matrix oracle, at the edges of their tiles
(8 and 32 q, 32 points, 64 and 128 curves) and of their dispatch rules.
"""

import numpy as np
import pytest

from oracle import resolution_ref


def _grid(nq, shuffle=False):
    q = np.linspace(0.01, 0.3, nq) if nq > 1 else np.array([0.05])
    qc = np.linspace(0.004, 0.4, 3*nq + 40)
    if shuffle:
        np.random.default_rng(1).shuffle(q)
    return q, qc


@pytest.mark.parametrize("length, width", [(0.05, 0.0), (0.05, 0.004), (0.02, 0.05)])
def test_slit_bands_hold_the_matrix(length, width):
    """The host's bands hold every nonzero weight of the dense slit matrix."""
    from sasmodels_b200.resolution import Slit1D
    q, qc = _grid(60)
    r = Slit1D(q, q_length=length, q_width=width, q_calc=qc)
    W = resolution_ref.slit_matrix(r._signed_q_calc, q, r._length, r._width)
    lo, hi = r._bands()
    for i in range(len(q)):
        nz = np.flatnonzero(W[:, i])
        assert nz[0] >= lo[i] and nz[-1] < hi[i]


@pytest.mark.gpu
@pytest.mark.parametrize("nq, sets, shuffle", [(1, 1, False), (31, 3, False), (33, 64, True),
                                               (200, 129, False), (257, 400, False),
                                               (700, 65, True), (1000, 1300, False)])
def test_band_apply_matches_matrix(cuda, nq, sets, shuffle):
    """One curve, few and many, against the dense matrix (the 1e-12 bar of the
    smearing tests), with rows of theory wider than the grid."""
    import torch
    from sasmodels_b200.resolution import Pinhole1D
    q, qc = _grid(nq, shuffle)
    r = Pinhole1D(q, 0.05*q, q_calc=qc)
    rng = np.random.default_rng(nq)
    th = rng.uniform(0.5, 2.0, (sets, len(qc) + 3))
    dev = torch.as_tensor(th, device="cuda")[:, :len(qc)]
    out = r.apply_sets(dev, torch.cuda.current_stream()).cpu().numpy()
    want = th[:, :len(qc)] @ r.weight_matrix
    np.testing.assert_allclose(out, want, rtol=1e-12, atol=0)
    one = r.apply(dev[0].contiguous()).cpu().numpy()
    np.testing.assert_allclose(one, want[0], rtol=1e-12, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("nq, sets", [(15, 1000), (16, 1000), (17, 1025), (31, 500), (33, 479),
                                      (500, 31), (500, 33), (875, 16), (875, 17)])
def test_many_curves_at_the_tile_edges(cuda, nq, sets):
    """Just beyond the rule for many curves, at the edges of its tiles of 16 and
    32 q and 8, 16 and 32 curves; each curve's result is its own."""
    import torch
    from sasmodels_b200.resolution import Pinhole1D
    assert 14000 <= nq*sets < 18000
    q, qc = _grid(nq)
    r = Pinhole1D(q, 0.05*q, q_calc=qc)
    th = np.random.default_rng(nq).uniform(0.5, 2.0, (sets, len(qc)))
    th[sets//2, len(qc)//2] = np.nan
    got = r.apply_sets(torch.as_tensor(th, device="cuda"),
                       torch.cuda.current_stream()).cpu().numpy()
    th[sets//2, len(qc)//2] = 0.0
    want = th @ r.weight_matrix
    sees = (r.band_lo <= len(qc)//2) & (len(qc)//2 < r.band_hi)
    want[sets//2, sees] = np.nan
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("sets", [1, 700])
def test_infinite_theory_reaches_only_its_bands(cuda, sets):
    """A point where a model is undefined spoils the q that see it, no other."""
    import torch
    from sasmodels_b200.resolution import Pinhole1D
    q, qc = _grid(200)
    r = Pinhole1D(q, 0.05*q, q_calc=qc)
    at = len(qc)//2
    th = torch.ones((sets, len(qc)), dtype=torch.float64, device="cuda")
    th[:, at] = float("inf")
    out = r.apply_sets(th, torch.cuda.current_stream()).cpu().numpy()
    sees = (r.band_lo <= at) & (at < r.band_hi)
    assert sees.any() and not sees.all()
    assert (np.isfinite(out) == ~sees[None, :]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("length, width", [(0.05, 0.0), (0.05, 0.004), (0.0, 0.0)])
@pytest.mark.parametrize("nq", [2, 31, 250])
def test_slit_plan_matches_formed_weights(cuda, monkeypatch, nq, length, width):
    """The plan against the kernel that forms the weights in every call."""
    from sasmodels_b200 import resolution as R
    q, qc = _grid(nq)
    qc = np.union1d(q, qc)
    th = np.random.default_rng(3).uniform(0.5, 2.0, len(qc))
    a = R.Slit1D(q, q_length=length, q_width=width, q_calc=qc).apply(th)
    monkeypatch.setattr(R, "MAX_WEIGHTS", -1)
    b = R.Slit1D(q, q_length=length, q_width=width, q_calc=qc).apply(th)
    np.testing.assert_allclose(a, b, rtol=1e-12, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("nq", [1, 511, 513, 1000])
@pytest.mark.parametrize("sets", [1, 4097])
def test_nllf_matches_numpy(cuda, nq, sets):
    """One curve and many; points of dy where 1/dy is not a normal number
    (their terms vanish) and an infinite theory value."""
    import torch
    from sasmodels_b200.resolution import nllf_sets
    rng = np.random.default_rng(nq)
    th = rng.uniform(0.5, 2.0, (sets, nq))
    y, dy = rng.uniform(0.5, 2.0, nq), rng.uniform(0.01, 0.1, nq)
    dy[::7] = 1e300
    th[-1, nq//2] = np.inf
    dy[nq//2] = 0.5
    got = nllf_sets(torch.as_tensor(th, device="cuda"), y, dy,
                    torch.cuda.current_stream()).cpu().numpy()
    want = 0.5*np.sum(((th - y)/dy)**2, axis=1)
    assert np.isinf(got[-1])
    np.testing.assert_allclose(got[:-1], want[:-1], rtol=1e-12, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("nbins", [1, 7, 8, 9, 40, 48, 200])
@pytest.mark.parametrize("nq", [1, 63, 65, 4097])
def test_pinhole2d_average_keeps_the_order(cuda, nq, nbins):
    """The 2D average is numpy's axis-0 reduction bit for bit."""
    import torch
    from sasmodels_b200.resolution import _check, _lib
    rng = np.random.default_rng(nbins)
    th, w = rng.uniform(-1, 2, (nbins, nq)), rng.uniform(0.1, 1.0, nbins)
    d = [torch.as_tensor(a, device="cuda") for a in (th, w)]
    out = torch.empty(nq, dtype=torch.float64, device="cuda")
    _check(_lib().sasb200_pinhole2d_average(nq, nbins, d[0].data_ptr(), d[1].data_ptr(), 3.0,
                                            out.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream), "average")
    num = th[0]*w[0]
    for b in range(1, nbins):
        num = num + th[b]*w[b]
    np.testing.assert_array_equal(out.cpu().numpy(), num/3.0)
