"""
A theory value that is not finite reaches only the measured q whose slit covers
its bin, with the weights kept per object as with those formed in every call.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length, width, step", [(0.002, 0.06, 1e-4), (0.002, 0.06, 1e-3),
                                                 (0.05, 0.004, 1e-3), (0.03, 0.0, 1e-3),
                                                 (0.0, 0.0, 1e-3)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite_theory_stays_in_its_bins(cuda, monkeypatch, length, width, step, bad):
    """Gaps between the steps across the slit (a short length and a fine grid),
    none, no width, and neither length nor width; a bad value every 13 bins."""
    from sasmodels_b200 import resolution as R
    q = np.linspace(0.05, 0.2, 40)
    qc = np.union1d(q, np.arange(0.01, 0.3, step))
    results = []
    for limit in (R.MAX_WEIGHTS, -1):
        monkeypatch.setattr(R, "MAX_WEIGHTS", limit)
        r = R.Slit1D(q, q_length=length, q_width=width, q_calc=qc)
        th = np.random.default_rng(5).uniform(0.5, 2.0, len(r.q_calc))
        clean = r.apply(th)
        th[::13] = bad
        results.append((clean, r.apply(th)))
    kept, formed = results
    np.testing.assert_allclose(kept[0], formed[0], rtol=1e-12, atol=0)
    np.testing.assert_array_equal(np.isnan(kept[1]), np.isnan(formed[1]))
    np.testing.assert_array_equal(np.isinf(kept[1]), np.isinf(formed[1]))
    fine = np.isfinite(formed[1])
    np.testing.assert_allclose(kept[1][fine], formed[1][fine], rtol=1e-12, atol=0)
