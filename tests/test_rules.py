"""The library's decisions that need no GPU (csrc/rules.h), compiled for the host."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = """
#include "rules.h"
extern "C" int in_place(int type, int where, int device) { return aldic::memory_in_place(type, where, device); }
extern "C" void quotients(long long k, const double *n, const double *s, double *first, double *q) {
  for (long long i = 0; i < k; ++i) {
    first[i] = aldic::faithful_quotient(n[i], s[i], 1.0 / s[i]);
    q[i] = aldic::rounded_quotient(n[i], s[i], 1.0 / s[i]);
  }
}
extern "C" double variance(long long n, long long s, long long q) { return aldic::sample_variance(n, s, q); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "2d_aldic_b200", "csrc"),
                    str(d / "shim.cpp"), "-o", str(d / "rules.so")], check=True)
    lib = C.CDLL(str(d / "rules.so"))
    lib.variance.restype = C.c_double
    lib.variance.argtypes = [C.c_longlong] * 3
    return lib


@pytest.mark.parametrize("device", [0, 1, 7])
def test_only_its_own_memory_is_used_in_place(rules, device):
    host, pinned, dev, managed = 0, 1, 2, 3       # cudaMemoryType
    for where in range(-2, 8):                    # -2, -1: of no device
        assert not rules.in_place(host, where, device)
        assert not rules.in_place(pinned, where, device)
        assert rules.in_place(dev, where, device) == (where == device)
        assert rules.in_place(managed, where, device)


@pytest.mark.parametrize("n", [2, 59049, 30_000_000, 60_000_000, 2_000_000_000])
@pytest.mark.parametrize("values", [(1, 99), (98, 99), (7, 7)])
def test_variance_of_many_evaluation_counts(rules, n, values):
    """Half of the subsets took one number of evaluations, half the other: exact up to
    the last divisions' roundings also where n sum(v^2) has more than 63 bits."""
    a, b = values
    k = n // 2
    s, q = k * a + (n - k) * b, k * a * a + (n - k) * b * b
    want = Fraction(n * q - s * s, n * (n - 1))
    assert rules.variance(n, s, q) == pytest.approx(float(want), rel=4 * 2.0 ** -53, abs=0)


def test_quotient_by_a_known_divisor_is_rounded_correctly(rules):
    """Divisors and deviations as images have them, and those where the product with the
    reciprocal is furthest off: a significand near 2 under one just below it."""
    r = np.random.default_rng(0)
    k = 200_000
    edge = lambda: np.ldexp(np.float64(2) - r.integers(2, 1 << 20, k) * 2.0 ** -52, r.integers(-3, 15, k))
    s = np.concatenate([r.uniform(0.5, 3e4, k), edge(), edge(), np.sqrt(r.integers(1, 1 << 30, k) / 7.0)])
    n = np.concatenate([r.uniform(-7e4, 7e4, k), edge(), edge() * (1 - r.integers(1, 4, k) * 2.0 ** -52),
                        r.integers(-65535, 65536, k) / 3.0 + 0.1])
    n[2 * k:3 * k] = s[2 * k:3 * k] * (1 - r.integers(1, 200, k) * 2.0 ** -53)
    first, q = np.empty_like(n), np.empty_like(n)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    rules.quotients(C.c_longlong(n.size), p(n), p(s), p(first), p(q))
    np.testing.assert_array_equal(q, n / s)
    pick = np.concatenate([r.choice(n.size, 4000), np.argsort(-np.abs(n * (1.0 / s) - n / s))[:1000]])
    for i in pick:
        exact = Fraction(float(n[i])) / Fraction(float(s[i]))
        assert abs(Fraction(float(first[i])) - exact) < Fraction(float(np.spacing(abs(first[i]))))
