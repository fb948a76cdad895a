"""
What the surrogate's entry points refuse before anything reaches the GPU.
"""

import glob
import os
import re
from types import SimpleNamespace

import numpy as np
import pytest

from sasmodels_b200.surrogate import Surrogate, TrainingGraph, sample_sets


def _surrogate():
    """A surrogate whose network is never reached."""
    S = Surrogate.__new__(Surrogate)
    S.torch, S.net, S.gate = None, SimpleNamespace(device=None), None
    return S


@pytest.mark.parametrize("q_shape", [(9,), (11,), (0,), (10, 1), (1, 10), ()])
def test_iq_refuses_q_of_another_length(q_shape):
    """Shorter, longer and two-dimensional q against ten points."""
    cols = sample_sets(10, np.random.default_rng(0))
    cols.update(set=np.arange(10), q=np.full(q_shape, 0.1))
    with pytest.raises(ValueError, match="q has shape"):
        _surrogate().iq(cols)


def test_iq_refuses_q_without_points():
    cols = {k: v[:0] for k, v in sample_sets(1, np.random.default_rng(0)).items()}
    cols.update(set=np.zeros(0, int), q=np.full(3, 0.1))
    with pytest.raises(ValueError, match="q has shape"):
        _surrogate().iq(cols)


@pytest.mark.parametrize("place", [("cpu", "meta", "meta"), ("meta", "cpu", "meta"),
                                   ("meta", "meta", "cpu")])
def test_capture_refuses_a_data_set_elsewhere(place):
    """Features, their low halves or targets on another device than the network
    (here the meta device, which has no memory that a kernel could reach)."""
    import torch
    shapes = ((256, 16), (256, 16), (256,))
    types = (torch.bfloat16, torch.bfloat16, torch.float32)
    data = [torch.zeros(s, dtype=t, device=d) for s, t, d in zip(shapes, types, place)]
    net = SimpleNamespace(torch=torch, device=torch.device("meta"))
    with pytest.raises(ValueError, match="must be on"):
        TrainingGraph(net, *data, 128, 1e-3, 10, 0, 1, 0.9, 0.999, 1e-8)


def test_every_entry_of_the_library_has_a_caller():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with open(os.path.join(root, "sasmodels_b200", "csrc", "mlp.cu")) as f:
        entries = re.findall(r"^(?:int32_t|const char \*) ?(sasb200_\w+)\(", f.read(), re.M)
    calls = ""
    for path in (glob.glob(os.path.join(root, "sasmodels_b200", "*.py"))
                 + glob.glob(os.path.join(root, "tests", "*.py"))):
        with open(path) as f:
            calls += f.read()
    assert len(entries) > 15
    assert [e for e in entries if "." + e + "(" not in calls] == []
