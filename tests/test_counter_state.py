"""Contexts share a device, so the tensor-core counters may keep nothing there that outlives a launch:
an expired wait is recorded in a word of the context that launched, which no other context reads
or clears."""
import os
import re

import pytest

import tensorfim_b200 as tf

CSRC = os.path.join(os.path.dirname(os.path.abspath(tf.__file__)), "csrc")


@pytest.mark.parametrize("name", ["count_f4.cu", "count_pk.cu"])
def test_no_device_variables(name):
    with open(os.path.join(CSRC, name)) as f:
        src = re.sub(r"//.*", "", f.read())
    # a device variable is a __device__ declaration without a parameter list
    assert not re.search(r"__device__[^;{}()]*;", src)
    assert "cudaGetSymbolAddress" not in src and "FromSymbol" not in src
    assert src.count("atomicExch(a.status, 1)") >= 1
