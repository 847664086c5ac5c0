"""The slices that the launch-shape autotuner times its candidates on
(csrc/mpf_tune.h): a permutation of the batch in which every slice samples the
whole order, in chunks of neighbours."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

SOURCE = r"""
#include "mpf_tune.h"
extern "C" long long slice_of(long long n) { return mpf::tune_slice(n); }
extern "C" void dealt(long long n, long long* out) { for (long long i = 0; i < n; ++i) out[i] = mpf::tune_dealt(i, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    src, so = str(d / "tune.cpp"), str(d / "tune.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, PKG, "csrc"), src, "-o", so])
    L = C.CDLL(so)
    L.slice_of.argtypes, L.slice_of.restype = [C.c_longlong], C.c_longlong
    L.dealt.argtypes, L.dealt.restype = [C.c_longlong, C.c_void_p], None
    return L


# the smallest tuned batch, one more ray, both sides of a whole group of chunks, an ordinary and the largest ordered batch
@pytest.mark.parametrize("n", [1 << 17, (1 << 17) + 1, 135167, 135168, 1000000, 1 << 22])
def test_slices_sample_the_whole_order(lib, n):
    out = np.empty(n, dtype=np.int64)
    lib.dealt(n, out.ctypes.data)
    assert np.array_equal(np.sort(out), np.arange(n))
    s = lib.slice_of(n)
    assert 0 < s and 4 * s <= n < 4 * s + 4096
    for k in range(4):
        part = out[k * s:n if k == 3 else (k + 1) * s]
        share = np.histogram(part, bins=4, range=(0, n))[0] / part.size
        assert np.all(np.abs(share - 0.25) <= 0.05), (k, share)      # a chunk or the rest is below 4 % of a slice
        assert np.all(np.diff(part[:s].reshape(-1, 32), axis=1) == 1)    # a warp's rays are neighbours
