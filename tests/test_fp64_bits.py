"""The float64 operations on integer bits (csrc/mpf_fp64.cuh) against the plain
operations, compiled for the host: zeros, subnormals, both ends of every range,
infinities and NaN of both signs, and seeded random operands.  Bits are equal,
NaN for NaN."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

SHIM = r"""
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
template <class T, class F> inline T bits_as(F f) { T t; std::memcpy(&t, &f, sizeof(t)); return t; }
inline unsigned __float_as_uint(float v) { return bits_as<unsigned>(v); }
inline long long __double_as_longlong(double v) { return bits_as<long long>(v); }
inline double __longlong_as_double(long long v) { return bits_as<double>(v); }
inline int __double2hiint(double v) { return (int)(__double_as_longlong(v) >> 32); }
inline int __double2loint(double v) { return (int)(__double_as_longlong(v) & 0xffffffffll); }
inline double __hiloint2double(int h, int l)
{
    return __longlong_as_double((long long)(((unsigned long long)(unsigned)h << 32) | (unsigned)l));
}
inline float __double2float_rn(double v) { return (float)v; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
"""

SOURCE = r"""
#include "mpf_fp64.cuh"
using namespace mpf;
#define EACH(name, T, R, bits, plain) \
    extern "C" void name(long long n, const T* a, const double* b, R* x, R* y) \
    { for (long long i = 0; i < n; ++i) { x[i] = (R)(bits); y[i] = (R)(plain); } }
EACH(t_wide, float, double, wide(a[i]), (double)a[i])
EACH(t_round32, double, double, round32(a[i]), (double)(float)a[i])
EACH(t_times_pow2, double, double, times_pow2(a[i], (int)b[i]), std::ldexp(a[i], (int)b[i]))
EACH(t_less64, double, int, less64(a[i], b[i]), a[i] < b[i])
EACH(t_negative, double, int, negative(a[i]), a[i] < 0.0)
EACH(t_axis, double, unsigned long long, axis_coord_bits((int)b[i], a[i]), axis_coord((int)b[i], a[i]))
EACH(t_center, double, double, coord_center_bits((int)b[i], (uint64_t)a[i]), coord_center((int)b[i], (uint64_t)a[i]))
EACH(t_divide, double, double, divide_by(a[i], b[i], 1.0 / b[i]), a[i] / b[i])
"""


@pytest.fixture(scope="module")
def bits(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("fp64")
    for name, text in (("cuda_runtime.h", SHIM), ("t.cpp", SOURCE)):
        with open(str(d / name), "w") as f:
            f.write(text)
    so = str(d / "t.so")
    subprocess.check_call([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(d),
                           "-I", os.path.join(ROOT, PKG, "csrc"), str(d / "t.cpp"), "-o", so])
    L = C.CDLL(so)

    def both(name, a, b=None, out=np.float64):
        a = np.ascontiguousarray(a)
        b = np.zeros(a.shape) if b is None else np.ascontiguousarray(b, dtype=np.float64)
        x, y = np.empty(a.shape, dtype=out), np.empty(a.shape, dtype=out)
        f = getattr(L, name)
        f.argtypes = [C.c_longlong] + 4 * [C.c_void_p]
        f(a.size, a.ctypes.data, b.ctypes.data, x.ctypes.data, y.ctypes.data)
        if x.dtype == np.float64:
            assert np.array_equal(np.isnan(x), np.isnan(y))
            x, y = np.where(np.isnan(x), 0, x).view(np.uint64), np.where(np.isnan(y), 0, y).view(np.uint64)
        bad = np.flatnonzero(x != y)
        assert bad.size == 0, (name, a[bad[:4]], b[bad[:4]])
    return both


def doubles():
    """Every exponent with mantissas at its ends and around a float's last bit, both signs; specials; random bits."""
    m = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, 1 << 29, 3 << 28, (1 << 52) - (1 << 28),
                  (1 << 52) - (1 << 28) - 1, (1 << 52) - 1], dtype=np.uint64)
    e = np.arange(2048, dtype=np.uint64) << np.uint64(52)
    v = (e[:, None] | m[None, :]).ravel()
    v = np.concatenate([v, np.random.default_rng(1).integers(0, 1 << 63, 1 << 18, dtype=np.uint64)])
    return np.concatenate([v, v | np.uint64(1 << 63)]).view(np.float64)


def test_conversions(bits):
    f = np.concatenate([np.arange(256, dtype=np.uint32)[:, None] << np.uint32(23) | np.array([0, 1, 2, 0x400000, 0x7fffff], np.uint32),
                        np.random.default_rng(2).integers(0, 1 << 31, (1 << 14, 5), dtype=np.uint32)]).ravel()
    with np.errstate(all="ignore"):
        bits("t_wide", np.concatenate([f, f | np.uint32(1 << 31)]).view(np.float32))
        bits("t_round32", doubles())


@pytest.mark.parametrize("e", [-511, -30, -1, 0, 1, 30, 511])
def test_products_with_powers_of_two(bits, e):
    bits("t_times_pow2", doubles(), np.full(doubles().shape, float(e)))


def test_compares(bits):
    """less64 for numbers (of two zeros the negative one is the smaller, of no
    use to its callers); negative for every pattern, NaN of both signs too."""
    d = doubles()
    bits("t_negative", d, out=np.int32)
    d = d[~np.isnan(d) & (d != 0)]
    rng = np.random.default_rng(3)
    with np.errstate(over="ignore"):
        others = (rng.permutation(d), d, np.nextafter(d, np.inf), np.nextafter(d, -np.inf), np.zeros(d.shape))
    for other in others:
        ok = (other != 0) | (d != 0)
        bits("t_less64", d[ok], other[ok], out=np.int32)
        bits("t_less64", other[ok], d[ok], out=np.int32)


@pytest.mark.parametrize("level", [0, 1, 2, 3, 9, 20, 31, 32])
def test_coordinates(bits, level):
    rng = np.random.default_rng(level)
    cells = np.arange(-6, 7) * 2.0 ** (2 - level)
    x = np.concatenate([rng.uniform(-2, 2, 1 << 16), rng.uniform(-6, 6, 1 << 12), cells - 2, cells, 2 + cells,
                        [-2.0, 2.0, 0.0, -0.0, 1e-300, -1e-300, 1e9, -1e9, -np.inf, np.nan, -np.nan]])
    x = np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf)])
    x = x[~(x > 1e9)]
    lv = np.full(x.shape, float(level))
    bits("t_axis", x, lv, out=np.uint64)
    c = np.unique(np.concatenate([[0, 1, 2 ** level - 1], rng.integers(0, 2 ** level, 1 << 12)])).astype(np.float64)
    bits("t_center", c, np.full(c.shape, float(level)))


def test_quotients_by_a_rounded_reciprocal(bits):
    """Operands whose quotient, reciprocal and residuals stay in the normal range: box lengths and k components."""
    rng = np.random.default_rng(5)
    b = np.concatenate([10.0 ** rng.uniform(20, 30, 1 << 17), np.ldexp(1.0, np.arange(60, 100)), [9.293e25, 9.3e25]])
    a = rng.choice([-1, 1], b.shape) * 10.0 ** rng.uniform(-30, 12, b.shape)
    bits("t_divide", a, b)
    bits("t_divide", np.nextafter(b, 0), b)
    bits("t_divide", np.full(b.shape, 299792458.0), b)
