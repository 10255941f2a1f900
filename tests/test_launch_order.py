"""Kernels launched as programmatic dependents (launch_pdl) begin before the
kernel ahead of them on the stream has ended, so each waits in its first
statement, and reads nothing through pointers that let the compiler move a load
above that wait.  Read from the sources; needs no GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qusim_gb300", "csrc")


def sources():
    return {os.path.basename(p): open(p).read() for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def kernels():
    """name -> (parameters, first statement) of every __global__ definition."""
    out = {}
    head = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*(?:\([^()]*\)[^()]*)*\))*\)\s*)?"
                      r"(\w+)\s*\(([^)]*)\)\s*\{\s*([^;]*;)")
    for text in sources().values():
        for m in head.finditer(text):
            out[m.group(1)] = (m.group(2), m.group(3))
    return out


def dependents():
    """Names of the kernels that launch_pdl launches, directly or through `auto k = name<...>`."""
    names = set()
    for text in sources().values():
        for m in re.finditer(r"launch_pdl\((\w+)", text):
            if m.group(1) != "k":
                names.add(m.group(1))
                continue
            names.add(re.findall(r"auto k = (\w+)", text[:m.start()])[-1])
    return sorted(names - {"void"})


def test_every_launch_is_found():
    defined = kernels()
    assert len(dependents()) >= 20
    assert not [n for n in dependents() if n not in defined]


@pytest.mark.parametrize("name", dependents())
def test_dependent_kernel_waits_first(name):
    assert kernels()[name][1] == "pdl_wait();"


@pytest.mark.parametrize("name", dependents())
def test_dependent_kernel_takes_no_restrict_pointer(name):
    assert "__restrict__" not in kernels()[name][0]
