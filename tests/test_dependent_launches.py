"""Kernels launched while the kernel before them still runs (griddepcontrol.wait, wait.cuh): what they
take from it is not declared constant for their lifetime."""
from __future__ import annotations

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "glu_public_b200",
                    "csrc")
# template parameters aside, a kernel: name, parameters, body up to the brace in the first column
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\([^\n]*?\)\s+)?(k_\w+)\(([^{]*?)\)\s*\{(.*?)\n\}",
                    re.S)


def kernels(name):
    with open(os.path.join(CSRC, name)) as f:
        return KERNEL.findall(f.read())


@pytest.mark.parametrize("name", ["kernels.cu", "dense.cu", "trsv.cu"])
def test_values_are_not_read_as_constants(name):
    """The plan's arrays are integers; doubles are values some kernel writes."""
    dependent = [(k, args) for k, args, body in kernels(name) if "after_previous()" in body]
    assert dependent
    for kernel, args in dependent:
        assert not re.search(r"const\s+(double|float)2?\s*\*\s*__restrict__", args), kernel


def test_every_dependent_launch_waits():
    """launch_next is for kernels that wait for the one before them on every path."""
    waits = {k for n in ("kernels.cu", "dense.cu", "trsv.cu") for k, _, body in kernels(n)
             if "after_previous()" in body}
    launched = set()
    for n in ("kernels.cu", "dense.cu", "trsv.cu"):
        with open(os.path.join(CSRC, n)) as f:
            launched |= set(re.findall(r"launch(?:_next)?\((k_\w+)", f.read()))
    assert launched and launched <= waits, launched - waits
