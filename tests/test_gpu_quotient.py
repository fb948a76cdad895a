"""
The quotient by a kept reciprocal (csrc/resolution.cu) is the division, bit for bit,
and the objective of one curve, few and many at the sizes where its kernels change.
"""

import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _quotients(x, d):
    """x[s, i]/d[i] by band_apply_sets: bands of one point of weight 1 and norm d."""
    import torch
    from sasmodels_b200.resolution import _check, _lib
    sets, nq = x.shape
    i32 = dict(dtype=torch.int32, device="cuda")
    lo = torch.arange(nq, **i32)
    hi, off = lo + 1, lo.to(torch.int64)
    w = torch.ones(nq, dtype=torch.float64, device="cuda")
    out = torch.empty_like(x)
    _check(_lib().sasb200_band_apply(
        sets, nq, nq, lo.data_ptr(), hi.data_ptr(), off.data_ptr(), w.data_ptr(), d.data_ptr(),
        x.data_ptr(), nq, out.data_ptr(), nq,
        ct.c_void_p(torch.cuda.current_stream().cuda_stream)), "band_apply")
    return out


@pytest.mark.parametrize("x_exp, d_exp", [((0, 0), (0, 0)), ((-20, 20), (-20, 20)),
                                          ((-1074, -900), (-60, 60)), ((-300, 300), (900, 963)),
                                          ((-1074, -1000), (900, 1023)),
                                          ((900, 1023), (-1074, -900)), ((0, 0), (-1074, 1023))])
def test_quotient_is_the_division(cuda, x_exp, d_exp):
    """Random significands and those next to 1 and 2; numerators, quotients and
    divisors down to the smallest number and up to the largest, and beyond."""
    import torch
    rng = np.random.default_rng(abs(x_exp[0]) + d_exp[1])

    def draw(shape, e):
        m = rng.uniform(1.0, 2.0, shape)
        edge = rng.integers(0, 4, shape)
        ulps = rng.integers(0, 4, shape)*2.0**-52
        m = np.where(edge == 0, 1.0 + ulps, np.where(edge == 1, 2.0 - 2.0**-52 - ulps, m))
        return np.ldexp(m, rng.integers(e[0], e[1] + 1, shape))*rng.choice([-1.0, 1.0], shape)
    nq, sets = 1000, 4000
    x = torch.as_tensor(draw((sets, nq), x_exp), device="cuda")
    d = torch.as_tensor(draw(nq, d_exp), device="cuda")
    x[::7, ::3] = 0.0
    assert torch.equal(_quotients(x, d), x/d)


@pytest.mark.parametrize("nq", [1, 255, 256, 257, 1000])
@pytest.mark.parametrize("sets", [1, 2, 1200, 1201, 1209])
def test_objective_of_finite_curves(cuda, nq, sets):
    """A block per curve (up to 1200) and a warp per curve, all curves compared."""
    import torch
    from sasmodels_b200.resolution import nllf_sets
    rng = np.random.default_rng(nq + sets)
    th = rng.uniform(0.5, 2.0, (sets, nq))
    y, dy = rng.uniform(0.5, 2.0, nq), rng.uniform(0.01, 0.1, nq)
    got = nllf_sets(torch.as_tensor(th, device="cuda"), y, dy,
                    torch.cuda.current_stream()).cpu().numpy()
    want = 0.5*np.sum(((th - y)/dy)**2, axis=1)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)


@pytest.mark.parametrize("sets", [1, 1201])
def test_objective_of_curves_that_are_not_finite(cuda, sets):
    import torch
    from sasmodels_b200.resolution import nllf_sets
    for bad in (np.inf, -np.inf, np.nan):
        th = np.ones((sets, 40))
        th[-1, 17] = bad
        got = nllf_sets(torch.as_tensor(th, device="cuda"), np.zeros(40), np.ones(40),
                        torch.cuda.current_stream()).cpu().numpy()
        assert np.all(got[:-1] == 20.0)
        assert np.isnan(got[-1]) if np.isnan(bad) else np.isposinf(got[-1])
