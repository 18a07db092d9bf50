"""The h solve's quotients by a kept reciprocal (csrc/divby.cuh) are those of
the division, bit for bit: the header's own code, compiled for the CPU, against
the CPU's division over the solve's arguments, u = 2 r / w in any unit of
length and the divisors 3 and 24, on quotients at and around the midpoint of
two numbers, and down to the smallest arguments it is stated for."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudasph_b200", "csrc")
SRC = """
#include "divby.cuh"
extern "C" void div_many(long n, const double *a, const double *b, double *q) {
  for (long i = 0; i < n; i++) q[i] = sph::div_by(a[i], b[i], 1.0 / b[i]);
}
"""


@pytest.fixture(scope="module")
def div_many(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("divby")
    (d / "d.cpp").write_text(SRC)
    subprocess.run([gxx, "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", str(d / "d.cpp"), "-I", CSRC,
                    "-o", str(d / "d.so")], check=True)
    lib = C.CDLL(str(d / "d.so"))

    def run(a, b):
        a, b = np.broadcast_arrays(np.asarray(a, np.float64), np.asarray(b, np.float64))
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        q = np.empty_like(a)
        p = C.c_void_p
        lib.div_many(C.c_long(a.size), p(a.ctypes.data), p(b.ctypes.data), p(q.ctypes.data))
        return q, a / b
    return run


def _same(pair):
    q, ref = pair
    return np.array_equal(q.view(np.int64), ref.view(np.int64))


@pytest.mark.parametrize("seed", range(4))
def test_ranges_of_any_unit(div_many, seed):
    rs = np.random.default_rng(seed)
    n = 400_000
    w = 10.0 ** rs.uniform(-100, 100, n)
    r = w * rs.uniform(0, 1, n) ** rs.choice([1.0, 8.0, 40.0], n)
    assert _same(div_many(2 * np.sqrt(r * r), w))


def test_constant_divisors(div_many):
    rs = np.random.default_rng(5)
    x = np.concatenate([rs.uniform(0, 1, 400_000), [0.0, 1e-90, 5e-97]])  # x^3 / 3
    assert _same(div_many(x * x * x, 3.0))
    x = np.concatenate([rs.uniform(1, 2, 400_000), [1.0, 2.0]])  # x^6 / 24
    assert _same(div_many((x * x * x) * (x * x * x), 24.0))


def test_quotients_at_the_midpoints(div_many):
    """a = b (q + ulp / 2) to a few ulp of a on both sides"""
    rs = np.random.default_rng(9)
    n = 100_000
    b = 1 + rs.integers(0, 2 ** 52, n) * 2.0 ** -52
    b[:4] = [1.0, 2 - 2.0 ** -52, 1 + 2.0 ** -52, 1.5]
    m = rs.integers(2 ** 52, 2 ** 53, n)
    a0 = np.array([float((int(x * 2 ** 52) * (2 * int(y) + 1)) >> 1) for x, y in zip(b, m)]) * 2.0 ** -104
    for k in range(-3, 4):
        a = a0 + k * np.spacing(a0)
        assert _same(div_many(a, b))
        assert _same(div_many(a, b * 2.0 ** 300)) and _same(div_many(a * 2.0 ** -500, b))


def test_smallest_arguments(div_many):
    rs = np.random.default_rng(3)
    a = 10.0 ** rs.uniform(-290, -200, 200_000)
    assert _same(div_many(a, rs.uniform(0.5, 30, a.size)))
    assert _same(div_many(np.zeros(3), np.array([1e-30, 3.0, 1e30])))
