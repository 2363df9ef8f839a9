"""The integer conversions of the vector kernels (convert.cuh), compiled for the
host: widen and narrow bit for bit against numpy, split_pair and PairSum against
exact sums, over every exponent, ties, subnormals, zeros, infinities and NaN."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
static float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static long long __double_as_longlong(double d) { long long u; std::memcpy(&u, &d, 8); return u; }
static double __hiloint2double(int hi, int lo) {
    const uint64_t u = (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
    double d; std::memcpy(&d, &u, 8); return d;
}
static float __fmul_rn(float a, float b) { return a * b; }
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
#include "convert.cuh"
extern "C" void widen_n(int n, const float* a, double* b) { for (int i = 0; i < n; ++i) b[i] = mg::widen(a[i]); }
extern "C" void narrow_n(int n, const double* a, float* b) { for (int i = 0; i < n; ++i) b[i] = mg::narrow(a[i]); }
extern "C" void split_n(int n, const double* a, float* h, float* l) {
    for (int i = 0; i < n; ++i) mg::split_pair(a[i], h[i], l[i]);
}
extern "C" void sum_n(int n, int m, const float* h, const float* l, double* s) {
    for (int i = 0; i < n; ++i) {
        mg::PairSum p;
        for (int k = 0; k < m; ++k) p.add(h[i * m + k], l[i * m + k]);
        s[i] = p.value();
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("conv")
    src, so = d / "conv.cpp", d / "conv.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "multigrid-ldg_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    return C.CDLL(str(so))


def call(f, *arrays, ints):
    f(*ints, *[a.ctypes.data_as(C.c_void_p) for a in arrays])


def same(a, b):
    """bit for bit, any NaN equal to any NaN"""
    u = np.uint32 if a.dtype == np.float32 else np.uint64
    return ((a.view(u) == b.view(u)) | (np.isnan(a) & np.isnan(b))).all()


def floats():
    rng = np.random.default_rng(1)
    edge = np.array([0, 1, 2, 0x7fffff, 0x800000, 0x800001, 0x3f800000, 0x7f7fffff, 0x7f800000, 0x7f800001, 0x7fc00000],
                    np.uint32)
    exps = (np.arange(256, dtype=np.uint32)[:, None] << 23 | np.array([0, 1, 0x400000, 0x7fffff], np.uint32)).ravel()
    u = np.concatenate([edge, exps, rng.integers(0, 2**31, 1000000, dtype=np.uint32)])
    return np.concatenate([u, u | np.uint32(0x80000000)]).view(np.float32)


def doubles():
    """random patterns, and for every exponent near FP32's range mantissas on and beside FP32 ties"""
    rng = np.random.default_rng(2)
    m = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, 1 << 29, 3 << 28, (3 << 28) - 1,
                  (1 << 52) - 1, (1 << 52) - (1 << 28), (1 << 52) - (1 << 28) - 1, (1 << 52) - (1 << 29)], np.uint64)
    exps = (np.arange(800, 1300, dtype=np.uint64)[:, None] << np.uint64(52) | m).ravel()
    near = rng.integers(850, 1200, 1000000).astype(np.uint64) << np.uint64(52) | rng.integers(0, 2**52, 1000000,
                                                                                             dtype=np.uint64)
    edge = np.array([0, 1, 0x000fffffffffffff, 0x0010000000000000, 0x7fefffffffffffff, 0x7ff0000000000000,
                     0x7ff0000000000001, 0x7ff8000000000000], np.uint64)
    u = np.concatenate([edge, exps, near, rng.integers(0, 2**63, 200000, dtype=np.uint64)])
    return np.concatenate([u, u | np.uint64(1 << 63)]).view(np.float64)


def test_widen(lib):
    a = floats()
    b = np.empty(len(a))
    call(lib.widen_n, a, b, ints=(len(a),))
    with np.errstate(invalid="ignore"):
        assert same(b, a.astype(np.float64))


def test_narrow(lib):
    a = doubles()
    b = np.empty(len(a), np.float32)
    call(lib.narrow_n, a, b, ints=(len(a),))
    with np.errstate(over="ignore", invalid="ignore"):
        assert same(b, a.astype(np.float32))


def test_split_pair(lib):
    """inside 2^-60 .. 2^100: h within half a unit of v (either side of a tie),
    h + l within 2^-48 of it; outside: the conversions"""
    v = doubles()
    h, l = np.empty(len(v), np.float32), np.empty(len(v), np.float32)
    call(lib.split_n, v, h, l, ints=(len(v),))
    with np.errstate(over="ignore", invalid="ignore"):
        h0 = v.astype(np.float32)
        l0 = (v - h0.astype(np.float64)).astype(np.float32)
    mag = np.abs(v)
    mid = (mag >= 2.0**-60) & (mag < 2.0**100)
    assert same(h[~mid], h0[~mid]) and same(l[~mid], l0[~mid])
    h, l, v = h[mid].astype(np.float64), l[mid].astype(np.float64), v[mid]
    ulp = 2.0 ** (np.floor(np.log2(np.abs(v))) - 23)
    assert (np.abs(v - h) <= 0.5 * ulp).all()
    assert (np.abs((v - h) - l) <= 2.0**-48 * np.abs(v)).all()


def test_pair_sum(lib):
    """PairSum.value() against the exact sum, terms of mixed size and sign: 2^-52
    of the result's own rounding and 2^-66 of the sum of magnitudes"""
    rng = np.random.default_rng(3)
    n, m = 2000, 27
    h = (rng.standard_normal((n, m)) * 2.0 ** rng.integers(-30, 30, (n, m))).astype(np.float32)
    l = (h * 2.0**-25 * rng.uniform(-1, 1, (n, m))).astype(np.float32)
    s = np.empty(n)
    call(lib.sum_n, np.ascontiguousarray(h), np.ascontiguousarray(l), s, ints=(n, m))
    for i in range(n):
        terms = [Fraction(float(x)) for x in np.concatenate([h[i], l[i]])]
        exact, size = sum(terms), sum(abs(t) for t in terms)
        assert abs(Fraction(float(s[i])) - exact) <= abs(exact) * Fraction(2)**-52 + size * Fraction(2)**-66
