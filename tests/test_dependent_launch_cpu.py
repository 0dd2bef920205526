"""Kernels of dependent launches (they call nb_grid_wait) start while the kernel before them still writes
what they read. The compiler turns loads through const __restrict__ parameters into read-only loads, which
ask for memory that nothing writes while the kernel runs and need not stay behind the wait; so these
kernels have no such parameters, and no read-only loads written out."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "n-body-simulation_gb300", "csrc")


def kernels():
    """(file, name, parameters, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__ void\s+(?:__\w+__\([^)]*\)\s*)*(\w+)\(([^{;]*)\)\s*\{", text):
            depth, k = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[k], 0)
                k += 1
            yield os.path.basename(path), m.group(1), m.group(2), text[m.end():k]


DEPENDENT = [k for k in kernels() if "nb_grid_wait" in k[3]]


def test_the_kernels_are_found():
    assert len(list(kernels())) > 40 and len(DEPENDENT) >= 18


@pytest.mark.parametrize("kernel", DEPENDENT, ids=lambda k: k[1])
def test_no_read_only_loads(kernel):
    _, _, parameters, body = kernel
    assert not re.search(r"const [^,]*__restrict__", parameters)
    assert "__ldg(" not in body and "ld.global.nc" not in body
    assert not re.search(r"\bload_(rec32|fix)(?!<false>)\b", body)
