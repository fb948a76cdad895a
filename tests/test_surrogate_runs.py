"""
The surrogate's evaluation of points in runs of equal parameters (features_runs,
finish_runs in csrc/mlp.cu) against the column features and numpy.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[1], [1, 1], [300], [5, 128, 1, 700, 3], [1]*257, [50000, 7]])
def test_device_eval_of_runs(cuda, lengths):
    """One point, one run, many single points, tiles split between runs; some
    sets outside the domain and a gate that rejects about half."""
    from sasmodels_b200.surrogate import MLP, Surrogate, sample_sets
    rng = np.random.default_rng(len(lengths))
    sets = sample_sets(len(lengths), rng)
    sets["radius"][::3] = 400.0
    sets["contrast"][1::5] = 0.0
    cols = {k: np.repeat(np.asarray(v), lengths) for k, v in sets.items()}
    n = sum(lengths)
    cols["q"] = np.exp(rng.uniform(np.log(5e-4), np.log(0.6), n))
    cols["set"] = np.repeat(np.arange(len(lengths)), lengths)
    S = Surrogate(seed=2)
    S.gate = MLP(seed=3, stream=S.net.stream)
    S.y_mean, S.y_std, S.g_mean, S.g_std = -1.0, 1.3, 0.2, 0.7
    with np.errstate(divide="ignore"):
        logi, g = S._outputs(cols)
    S.cal_tols, S.cal_thresh = np.array([1e-3]), np.array([np.exp(np.median(g))])
    I, accept = S._device_eval(cols, 0.01)
    assert I.shape == accept.shape == (n,) and accept.dtype == bool
    # exp amplifies a rounding of its argument (|log I| < 40) to 40 ulp
    np.testing.assert_allclose(I, np.exp(logi), rtol=1e-13, atol=0)
    want = S.inside(cols) & (g <= np.log(S.cal_thresh[0]))
    np.testing.assert_array_equal(accept, want)
    # nothing is trusted without a calibration
    S.cal_thresh = None
    assert not S._device_eval(cols, 0.01)[1].any()
    I0, a0 = S._device_eval({k: v[:0] for k, v in cols.items()}, 0.01)
    assert I0.shape == a0.shape == (0,)
