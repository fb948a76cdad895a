"""
Kernels that may be resident while those before them on the stream still write
(csrc/tc_ptx.cuh, dependency_wait) must not promise that their inputs never change.
"""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sasmodels_b200", "csrc")


def _dependent_kernels():
    """(name, signature, body) of the kernels that wait for those before them."""
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "mlp*.cu*"))):
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for part in text.split("__global__")[1:]:
            if "dependency_wait()" in part:
                head, body = part.split("{", 1)
                found.append((re.findall(r"(\w+)\(", head)[-1], head, body))
    return found


def test_the_dependent_kernels_are_seen():
    names = {name for name, _, _ in _dependent_kernels()}
    assert {"mlp_serve", "mlp_halves", "mlp_backward_t", "mlp_weight_grads", "adam_pack"} <= names


@pytest.mark.parametrize("name, head, body", _dependent_kernels(),
                         ids=[k[0] for k in _dependent_kernels()])
def test_no_read_only_promise(name, head, body):
    assert not re.search(r"const\s+\w+\s*\*\s*(const\s*)?__restrict__", head), name
    assert "__ldg(" not in body and "ld.global.nc" not in body, name
