"""The powers and quotients of the EAM pair functions (sg_pairmath.h, compiled here for the host: the same
IEEE operations as on the device) against exact ones: quotients by a shared reciprocal against the
division, 19th and 20th powers against extended precision, and both past the arguments of a pair."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "surfacegrowthconsole_gb300" / "csrc"
N = 1 << 17

SOURCE = r"""
#include "sg_pairmath.h"
extern "C" void powers(const float *x, float *p, float *q, float *r, int n) {
  for (int i = 0; i < n; i++) {
    sg::pow19and20(x[i], p[i], q[i]);
    r[i] = sg::pow20(x[i]);
  }
}
extern "C" void exact(const float *x, long double *p, long double *q, int n) {
  for (int i = 0; i < n; i++) {
    const long double a = x[i], a2 = a * a, a4 = a2 * a2, a16 = a4 * a4 * a4 * a4;
    p[i] = a16 * a2 * a;
    q[i] = a16 * a4;
  }
}
extern "C" void quotients(const float *a, const float *b, float *q, int n) {
  for (int i = 0; i < n; i++) q[i] = sg::divBy(a[i], b[i], 1.f / b[i]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairmath")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(CSRC), "-o",
                    str(d / "m.so"), str(d / "m.cpp")], check=True)
    return C.CDLL(str(d / "m.so"))


def ptr(x):
    return x.ctypes.data_as(C.c_void_p)


def powers(lib, x):
    x = np.ascontiguousarray(x, np.float32)
    p, q, r = (np.empty_like(x) for _ in range(3))
    lib.powers(ptr(x), ptr(p), ptr(q), ptr(r), len(x))
    return p, q, r


def divide(lib, a, b):
    a, b = (np.ascontiguousarray(z, np.float32) for z in (a, b))
    q = np.empty_like(a)
    lib.quotients(ptr(a), ptr(b), ptr(q), len(a))
    with np.errstate(over="ignore", invalid="ignore"):
        return q, a / b


def same(x, y):
    return np.array_equal(np.where(np.isnan(x), np.float32(0), x).view(np.int32),
                          np.where(np.isnan(y), np.float32(0), y).view(np.int32)) and np.array_equal(np.isnan(x), np.isnan(y))


def denominators(lib, x):
    return np.minimum(np.float32(1) + powers(lib, x)[1], np.float32(8e37))


def arguments(rng, top):
    """x of either sign, evenly spread and over its logarithm, with the ends."""
    x = np.concatenate([rng.uniform(-top, top, N), np.exp(rng.uniform(np.log(1e-6), np.log(top), N)) * rng.choice([-1, 1], N),
                        [0.0, -0.0, 1.0, -1.0, top, -top, 1e-30]])
    return x.astype(np.float32)


@pytest.mark.parametrize("top", [2.3, 63.99])
def test_powers(lib, top):
    """x^19 and x^20 within 0.501 of a unit in the last place down to 2^-110, within 2 to the smallest normal
    number."""
    x = arguments(np.random.RandomState(1), top)
    p, q, r = powers(lib, x)
    assert same(q, r)
    e19, e20 = np.empty(len(x), np.longdouble), np.empty(len(x), np.longdouble)
    lib.exact(ptr(x), ptr(e19), ptr(e20), len(x))
    for got, want in ((p, e19), (q, e20)):
        for least, bound in ((-110, 0.501), (-126, 2.0)):
            above = np.abs(want) >= np.longdouble(2.0) ** least
            ulp = np.longdouble(2.0) ** (np.floor(np.log2(np.abs(want[above]))) - 23)
            assert (np.abs(got[above] - want[above]) / ulp).max() <= bound
        # below them: a few of the smallest units
        assert np.abs(got[~above] - want[~above]).max() <= 4 * np.longdouble(2.0) ** -149


def test_powers_past_the_pairs_range(lib):
    x = np.array([64, -64, 80, 84.3, -84.3, 90, 1e10, -1e10, np.inf, -np.inf, np.nan], np.float32)
    p, q, r = powers(lib, x)
    with np.errstate(over="ignore"):
        w19, w20 = (x.astype(np.float64) ** k for k in (19, 20))
        big = np.abs(w20) >= 2.0 ** 128
        f19, f20 = w19.astype(np.float32), w20.astype(np.float32)
    assert same(q, r)
    for got, want in ((p, f19), (q, f20)):
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
        ok = np.isfinite(want)
        assert np.abs(got[ok] / want[ok] - 1).max() < 1e-6 and np.array_equal(np.sign(got[~np.isnan(got)]), np.sign(want[~np.isnan(want)]))
    assert big.any()


def test_quotients_are_the_division(lib):
    """By the pair functions' denominators, 1 + x^20 capped, for numerators whose quotient's remainder is a
    normal number: from 2^-100 times the denominator on."""
    rng = np.random.RandomState(2)
    for top in (2.3, 63.99):
        b = denominators(lib, arguments(rng, top))
        q, want = divide(lib, b * np.exp(rng.uniform(np.log(2.0 ** -76), 0, len(b))), b)
        assert same(q, want)
        q, want = divide(lib, rng.choice([-1, 1], len(b)) * np.exp(rng.uniform(np.log(1e-6), np.log(1e30), len(b))), b)
        lost = np.abs(want) < 2.0 ** -100
        assert same(q[~lost], want[~lost])
        assert np.abs(q[lost].astype(np.float64) - want[lost]).max(initial=0.0) <= 2.0 ** -123
    one = np.ones(1 << 16, np.float32)  # any numerator by 1
    a = np.arange(1 << 16, dtype=np.uint32).astype(np.uint32) * np.uint32(65521)
    a = a.view(np.float32)
    a = np.where(np.isfinite(a), a, np.float32(0))
    assert same(*divide(lib, a, one))


def test_the_pair_functions_own_quotients(lib):
    """20 x^19 / (1 + x^20) over every size of x that a pair within a cutoff has."""
    x = arguments(np.random.RandomState(3), 2.3)
    p, q, _ = powers(lib, x)
    got, want = divide(lib, np.float32(20) * p, np.float32(1) + q)
    assert same(got + np.float32(0), want + np.float32(0))  # but for the sign of a zero
