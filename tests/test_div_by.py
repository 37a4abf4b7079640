"""Division by a launch constant (csrc/icb_div.cuh) against the general
division, bit for bit (CPU: the header built with the host compiler, without
contraction; it uses IEEE operations only).  Divisors and dividends around the
ends of the ranges in which the corrected product is taken, zeros of both
signs, infinities, NaN, subnormals, and quotients as close to a rounding
boundary as 53-bit numbers allow."""
from __future__ import annotations

import ctypes as C
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "icarion_b200" / "csrc"

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __noinline__
static int __double2hiint(double a) { uint64_t u; std::memcpy(&u, &a, 8); return static_cast<int>(u >> 32); }
using std::fma;
#include "icb_div.cuh"
extern "C" void run(long n, const double* a, const double* b, double* got, double* want) {
    for (long i = 0; i < n; ++i) {
        got[i] = icb::div_by(a[i], b[i], icb::div_reciprocal(b[i]));
        volatile double x = a[i], y = b[i];
        want[i] = x / y;
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC", "-I", str(CSRC),
                    str(d / "shim.cpp"), "-o", str(d / "shim.so")], check=True)
    return C.CDLL(str(d / "shim.so"))


def _check(lib, a, b):
    a, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b))
    got, want = np.empty_like(a), np.empty_like(a)
    p = lambda v: v.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    lib.run(C.c_long(a.size), p(a), p(b), p(got), p(want))
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    bad = np.flatnonzero(~same)[:5]
    assert same.all(), [(a[i], b[i], got[i], want[i]) for i in bad]


def _around(exps, rng, n=40):
    """Numbers at, next to and above powers of two."""
    out = []
    for e in exps:
        v = np.ldexp(1.0, e)
        out += [v, np.nextafter(v, 0), np.nextafter(v, np.inf)] + list(np.ldexp(rng.uniform(1, 2, n), e))
    return np.array(out)


def test_range_edges_and_special_values(lib):
    rng = np.random.default_rng(1)
    b = _around([-1074, -1022, -301, -300, -299, -84, 0, 299, 300, 301, 302, 1023], rng)
    a = _around([-1074, -1022, -624, -623, -622, -300, 0, 1, 575, 576, 577, 578, 1023], rng)
    a = np.concatenate([a, [0.0, np.inf, np.nan]])
    b = np.concatenate([b, -b[:20], [0.0, -0.0, np.inf, -np.inf, np.nan]])
    A, B = np.meshgrid(a, b)
    _check(lib, A.ravel(), B.ravel())
    _check(lib, -A.ravel(), B.ravel())


def test_random_quotients(lib):
    rng = np.random.default_rng(2)
    n = 2_000_000
    a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-623, 577, n)) * rng.choice([-1.0, 1.0], n)
    b = np.ldexp(rng.uniform(1, 2, n), rng.integers(-300, 301, n))
    _check(lib, a, b)
    _check(lib, a[:1000] * b[:1000], b[:1000])           # (nearly) exact quotients


def test_quotients_next_to_a_rounding_boundary(lib):
    """A / B = (2 Q + 1) / 2^54 - r / (B 2^54) with 53-bit A, B, Q and small odd
    r: the quotient lies r / B of half a unit from a midpoint."""
    rnd = random.Random(3)
    a, b = [], []
    while len(a) < 40_000:
        B = rnd.randrange(1 << 52, 1 << 53) | 1
        r = rnd.choice([1, 3, 5, 7, -1, -3, -5, -7])
        q2 = r * pow(B, -1, 1 << 54) % (1 << 54)         # 2 Q + 1
        A = (q2 * B - r) >> 54
        if not (1 << 52) <= A < (1 << 53):
            continue
        assert q2 * B - r == A << 54
        a.append(float(A))
        b.append(float(B))
    a, b = np.array(a), np.array(b)
    for ea, eb in ((0, 0), (-600, 200), (500, -300), (-670, -352), (520, 247)):
        _check(lib, np.ldexp(a, ea), np.ldexp(b, eb))


def test_divisors_whose_reciprocal_rounds_worst(lib):
    """Divisors just below 2 (a reciprocal half a unit off just above 1/2) and
    quotients just below 2, where a y is furthest, 1.5 units, from a / b."""
    rng = np.random.default_rng(4)
    n = 2_000_000
    b = 2.0 - 2.0 ** -52 * rng.integers(1, 1 << 12, n)
    a = b * (2.0 - 2.0 ** -52 * rng.integers(1, 1 << 12, n))
    a = a + np.spacing(a) * rng.integers(-2, 3, n)
    _check(lib, a, b)
    _check(lib, a, np.full_like(a, np.nextafter(2.0, 0)))
