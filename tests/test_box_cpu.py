"""The entries that a tree build adds to its box (nb_fix.cuh, compiled as plain C++): they stay within
BOX_WORDS, which sizes the one-block build's shared copy and the tree's own, and are the centre, the
scale exponent K and the FP32 edge^2 of the box."""

import ctypes as C
import math
import os
import struct
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "nb_fix.cuh"
extern "C" int box_words() { return nbfix::BOX_WORDS; }
extern "C" void extras(double* box, unsigned i) { nbfix::box_extras(box, i); }
"""


@pytest.fixture(scope="module")
def fix(tmp_path_factory):
    d = tmp_path_factory.mktemp("box")
    (d / "box.cpp").write_text(SOURCE)
    so = str(d / "libbox.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "n-body-simulation_gb300", "csrc"), str(d / "box.cpp"), "-o",
                    so], check=True)
    lib = C.CDLL(so)
    lib.extras.argtypes = [C.POINTER(C.c_double), C.c_uint]
    return lib


@pytest.mark.parametrize("lo,hi", [((-1.0, -0.5, 0.0), (0.75, 2.0, 0.25)), ((0.0, 0.0, 0.0), (3e5, 1.0, 7.0)),
                                   ((-4.0, -4.0, -4.0), (4.0, 4.0, 4.0)),
                                   ((-1e-30, 0.0, 0.0), (1e-31, 1e-33, 1e-30))])
def test_entries_and_bounds(fix, lo, hi):
    words = fix.box_words()
    edge = max(h - l for l, h in zip(lo, hi))
    guard = 1234.5
    box = (C.c_double * (words + 16))(*([guard] * (words + 16)))
    for k, v in enumerate((*lo, *hi, edge)):
        box[k] = v
    for i in range(32):
        fix.extras(box, i)
    assert list(box[words:]) == [guard] * 16
    assert guard not in list(box[:words])
    assert list(box[7:10]) == [l + edge / 2 for l in lo]
    K = math.frexp(max(abs(v) for v in (*lo, *hi)))[1]  # the least with every |v| below 2^K
    assert box[10] == K
    low, high = struct.unpack("<Ii", struct.pack("<d", box[11]))
    with np.errstate(over="ignore", under="ignore"):
        want = np.array([np.float32(edge * edge)]).view(np.uint32)[0]
    assert (high, low) == (K, want)
