"""The rule of kernels that wait for their predecessor on the device (`pdl_begin`, csrc/common.cuh): nothing an earlier kernel may
have written is read through a pointer that lets the compiler move the load in front of the wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "socket_b200", "csrc")
KERNEL = re.compile(r"__global__ void __launch_bounds__\([^)]*\)\s+(\w+)\(([^{;]*?)\)\s*\{\s*(?://[^\n]*\n\s*)*pdl_begin\(\);", re.S)


def _kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            for m in KERNEL.finditer(f.read()):
                yield pytest.param(m[2], id=f"{os.path.basename(path)}:{m[1]}")


def test_the_kernels_are_found():
    assert len(list(_kernels())) >= 15


@pytest.mark.parametrize("params", list(_kernels()))
def test_inputs_are_not_restrict(params):
    assert not [p for p in params.split(",") if "const" in p and "__restrict__" in p]
