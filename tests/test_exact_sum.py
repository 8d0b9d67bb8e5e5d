"""The order-independent sum of the adjoint's upstream chains (exact_sum.cuh,
compiled for the host) against the exact rational sum: cancelling chains of either sign,
wide ranges of magnitude, subnormals, overflow, infinities and NaN."""

import ctypes
import math
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "up3d_b200" / "csrc"
SOURCE = """
#include "exact_sum.cuh"
extern "C" double chain(const double* v, int n) {
    int top = 0;
    for (int i = 0; i < n; ++i) top = up3d::exponent_field(v[i]) > top ? up3d::exponent_field(v[i]) : top;
    up3d::ExactSum s(top);
    for (int i = 0; i < n; ++i) s.add(v[i]);
    return s.value();
}
"""


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact_sum")
    (d / "chain.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "chain.cpp"), "-o",
                    str(d / "chain.so")], check=True)
    f = ctypes.CDLL(str(d / "chain.so")).chain
    f.restype, f.argtypes = ctypes.c_double, [ctypes.c_void_p, ctypes.c_int]

    def call(v):
        v = np.ascontiguousarray(v, dtype=np.float64)
        return f(v.ctypes.data, len(v))
    return call


def _chains(rng, n):
    yield rng.uniform(0.5, 1.0, n)
    yield -rng.uniform(0.5, 1.0, n)
    yield rng.standard_normal(n)
    yield rng.standard_normal(n) * 10.0 ** rng.integers(-12, 13, n)
    v = rng.standard_normal(n)                       # cancels but for the last bits
    yield np.append(v, -math.fsum(v) * (1.0 + rng.integers(-3, 4) * 2.0 ** -52))
    yield np.append(v, -math.fsum(v) * (1.0 - 2.0 ** -51))
    yield v * 2.0 ** -1060                           # subnormals
    yield v * 2.0 ** 1018


@pytest.mark.parametrize("n", [2, 3, 8, 31, 1000])
def test_sum_is_the_exact_one_rounded(chain, n):
    rng = np.random.default_rng(n)
    for v in _chains(rng, n):
        s, exact = chain(v), float(sum(map(Fraction, v)))
        # a term's rounding is 2^-96 of the largest, the result's half a unit
        assert abs(s - exact) <= len(v) * 2.0 ** -96 * np.abs(v).max() + np.spacing(abs(exact))
        assert chain(-v) == -s
        assert chain(rng.permutation(v)) == s and chain(v[::-1]) == s


@pytest.mark.parametrize("v", [(1.0, -1.0 - 2.0 ** -52), (1.0, -1.0 - 3 * 2.0 ** -52), (-1.0, 0.9999999999999),
                               (1e16, 1.0, -1e16), (1.0, 2.0 ** -80, -1.0), (5e-324, 5e-324, -1e-323)])
def test_cancellation_is_exact(chain, v):
    assert chain(v) == math.fsum(v) and chain([-x for x in v]) == -math.fsum(v)


def test_not_finite(chain):
    inf, nan = math.inf, math.nan
    assert chain([1.0, inf, -2.0]) == inf and chain([-inf, 1e308]) == -inf
    assert math.isnan(chain([inf, -inf, 1.0])) and math.isnan(chain([1.0, nan])) and math.isnan(chain([inf, nan]))
    assert chain([1.7e308, 1.7e308, 1.0]) == inf
    assert chain([1.7e308, 1.7e308, -1.7e308]) == 1.7e308     # no overflow on the way
    assert chain([0.0, -0.0]) == 0.0
