"""
Copies of a resolution object: the weights kept on the device belong to one object.
"""

import copy
import pickle

import numpy as np
import pytest

from sasmodels_b200.resolution import Pinhole1D, Slit1D

Q = np.linspace(0.01, 0.3, 30)
MAKERS = [lambda: Pinhole1D(Q, 0.05*Q), lambda: Slit1D(Q, q_length=0.05, q_width=0.004)]
COPIES = [copy.copy, copy.deepcopy, lambda r: pickle.loads(pickle.dumps(r))]


@pytest.mark.parametrize("make", MAKERS)
@pytest.mark.parametrize("copied", COPIES)
def test_copies_leave_the_device_state(make, copied):
    r = make()
    r._dev = dict(plan=dict(lo=4096))             # an address, as after an application
    c = copied(r)
    assert c._dev is None and r._dev["plan"]["lo"] == 4096
    np.testing.assert_array_equal(c.q_calc, r.q_calc)


@pytest.mark.gpu
@pytest.mark.parametrize("make", MAKERS)
@pytest.mark.parametrize("copied", COPIES)
def test_a_copy_outlives_its_original(cuda, make, copied):
    import torch
    r = make()
    theory = torch.rand(len(r.q_calc), dtype=torch.float64, device="cuda")
    want = r.apply(theory).clone()
    c = copied(r)
    del r
    torch.cuda.empty_cache()
    assert torch.equal(c.apply(theory), want)
