"""The traveltime sweeps' divisions by known divisors (csrc/kcig_div.h,
compiled for the host) against the machine's correctly rounded division, bit
for bit: FP32 over the whole range of dividends, at the ends of the quick
form's range and with divisors whose reciprocal is no normal number; FP64 over
the range the sweeps form."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kirch_datuming_b200", "csrc")
SOURCE = """
#include "kcig_div.h"
extern "C" void divide32(const float *a, const float *b, float *q, int n)
{
    for (int i = 0; i < n; i++) q[i] = kcig::div_by(a[i], kcig::div_prepare(b[i]));
}
extern "C" void divide64(const double *a, const double *b, double *q, int n)
{
    for (int i = 0; i < n; i++) q[i] = kcig::div_by(a[i], b[i], 1.0 / b[i]);
}
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "div.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "div.so"),
                    str(d / "div.cpp"), "-lm"], check=True)
    lib = ctypes.CDLL(str(d / "div.so"))

    def run(a, b):
        q = np.empty_like(a)
        f = lib.divide32 if a.dtype == np.float32 else lib.divide64
        f(*(v.ctypes.data_as(ctypes.c_void_p) for v in (a, b, q)), ctypes.c_int(a.size))
        return q
    return run


def _same(got, want):
    # bit for bit, but for the sign of a zero
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    u = np.uint32 if got.dtype == np.float32 else np.uint64
    bad = np.flatnonzero((got.view(u) != want.view(u)) & ~nan & ((got != 0) | (want != 0)))
    assert bad.size == 0, (bad.size, got[bad[:4]], want[bad[:4]])


def _floats(rng, n, lo, hi, dtype):
    v = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
    return v.astype(dtype)


@pytest.mark.parametrize("spacing", [1e-4, 0.0031, 0.01, 0.5, 0.7, 1.0, 6.25, 12.5, 333.0, 1e7, 1e19, 1e-19, 1e20, 1e-23])
def test_fp32_every_dividend(divide, spacing):
    rng = np.random.default_rng(3)
    d = np.float32(spacing)
    with np.errstate(all="ignore"):
        dd = d * d
        a = _floats(rng, 200000, -149, 128, np.float32)
        edges = np.float32([0.0, -0.0, np.inf, -np.inf, np.nan, 3.4028235e38, -3.4028235e38, 1e-45, 1.17549435e-38])
        near = [np.float32(2.0 ** e) * (1 + np.arange(-300, 300, dtype=np.float32) * np.float32(2 ** -23))
                for e in (-80, -126, 86, 126)]
        quot = [np.float32(2.0 ** e) * dd * (1 + np.arange(-300, 300, dtype=np.float32) * np.float32(2 ** -23))
                for e in (-126, -100, 126)]
        a = np.concatenate([a, edges, *near, *quot]).astype(np.float32)
        b = np.full_like(a, dd)
        _same(divide(a, b), a / b)


def test_fp32_every_divisor(divide):
    rng = np.random.default_rng(4)
    with np.errstate(all="ignore"):
        a, b = _floats(rng, 400000, -149, 128, np.float32), np.abs(_floats(rng, 400000, -149, 128, np.float32))
        ends = np.float32(2) ** rng.integers(-20, 20, 4000).astype(np.float32)
        b[:4000] = ends * np.nextafter(np.float32(2), np.float32(0))  # mantissas of ones
        a[:4000] = _floats(rng, 4000, -20, 20, np.float32)
        _same(divide(a, b), a / b)


def test_fp64_range_of_the_sweeps(divide):
    rng = np.random.default_rng(5)
    a = _floats(rng, 400000, -300, 420, np.float64)
    rdx = [np.abs(_floats(rng, 400000, -60, 60, np.float32)).astype(np.float64) * rng.choice([1.0, 2.25], 400000)
           for _ in range(2)]
    _same(divide(a, rdx[0]), a / rdx[0])
    both = rdx[0] + rdx[1]
    _same(divide(a, both), a / both)
    three = np.full_like(a, 3.0)
    _same(divide(a, three), a / three)
