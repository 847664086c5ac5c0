"""Which cell offsets lie in a stencil record (csrc/mpf_keys.cuh), compiled for
the host: -1, 0 and 1 along every axis and nothing else, at both ends of int
too, to which the conversion of a far point's offset saturates."""
import ctypes as C
import itertools
import os
import subprocess

import pytest

from conftest import PKG, ROOT

SOURCE = r"""
#include "mpf_keys.cuh"
extern "C" int within(int x, int y, int z) { return mpf::within_one_cell(x, y, z); }
"""


@pytest.fixture(scope="module")
def within(tmp_path_factory):
    d = tmp_path_factory.mktemp("near")
    src, so = str(d / "near.cpp"), str(d / "near.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, PKG, "csrc"), src, "-o", so])
    return C.CDLL(so).within


def test_only_the_27_cells_around(within):
    ends = [-2 ** 31, -2 ** 31 + 1, -2, -1, 0, 1, 2, 2 ** 31 - 2, 2 ** 31 - 1]
    for o in itertools.product(ends, repeat=3):
        assert bool(within(*o)) == all(-1 <= v <= 1 for v in o), o
