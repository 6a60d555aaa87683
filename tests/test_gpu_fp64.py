"""Reciprocals and quotients by Newton's iteration (csrc/fp64.hpp) over the exponents that the
factorisations and the posteriors accept, against extended precision."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.helpers import ROOT

pytestmark = pytest.mark.gpu

FAST_RECIPROCAL, RECIPROCAL, QUOTIENT, DIVIDE = range(4)
COUNT = 400000


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fp64") / "fp64.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call([f"{cuda}/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                           "-shared", "-Xcompiler", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "host", "fp64_test.cu")])
    fn = ctypes.CDLL(so).fp64_evaluate
    p = ctypes.c_void_p

    def call(op, x, n=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        n = np.ones_like(x) if n is None else np.ascontiguousarray(n, dtype=np.float64)
        out = np.empty_like(x)
        e = fn(op, ctypes.c_int64(len(x)), x.ctypes.data_as(p), n.ctypes.data_as(p), out.ctypes.data_as(p))
        assert e == 0, f"CUDA error {e}"
        return out

    return call


def values(seed, lo, hi):
    """Random mantissas over the exponents from lo to hi, the ends among them, and mantissas next to
    powers of two."""
    rng = np.random.default_rng(seed)
    e = rng.uniform(np.log2(lo), np.log2(hi), COUNT)
    m = 1 + rng.random(COUNT)
    m[:1000] = 1 + np.arange(1000) * 2.0 ** -52
    m[1000:2000] = 2 - np.arange(1, 1001) * 2.0 ** -52
    return np.clip(np.concatenate([np.ldexp(m, np.floor(e).astype(int)), [lo, hi, 1.0, 0.5, 2.0]]), lo, hi)


def ulps(got, exact):
    """Distance from the extended-precision value in units in the last place of its double."""
    unit = np.spacing(np.abs(exact.astype(np.float64)))
    return np.abs((got.astype(np.longdouble) - exact) / unit)


# Bounds: half a unit for the last rounding, and what the steps before leave: below 2^-20 units where
# nothing underflows; extended precision itself adds 2^-11.
HALF = 0.5 + 2.0 ** -10


def test_reciprocal_over_the_pivots_range(evaluate):
    x = values(1, 2.3e-308, 4e307)
    for sign in (1, -1):
        got = evaluate(FAST_RECIPROCAL, sign * x)
        assert ulps(got, sign / x.astype(np.longdouble)).max() <= HALF
        assert np.mean(got != evaluate(DIVIDE, sign * x)) < 1e-5


def test_reciprocal_of_any_value(evaluate):
    """The likelihoods' range and both its ends; zeros, NaN, infinities, negative and subnormal values as
    the division."""
    x = values(2, 0.9e-300, 1.1e300)
    assert ulps(evaluate(RECIPROCAL, x), 1 / x.astype(np.longdouble)).max() <= HALF
    x = np.array([0.0, -0.0, np.nan, np.inf, -np.inf, -1.5, 1e-300, 1e300, 5e-324, 1e-310, 1.7e308])
    np.testing.assert_array_equal(evaluate(RECIPROCAL, x), evaluate(DIVIDE, x))


def test_quotients_over_the_likelihoods_range(evaluate):
    """n / x for n of the size of x, as in a posterior (n <= 4 x)."""
    x = values(3, 1.001e-300, 0.999e300)
    n = x * np.random.default_rng(4).uniform(0, 4, len(x))
    got, exact = evaluate(QUOTIENT, x, n), n.astype(np.longdouble) / x
    assert ulps(got, exact).max() <= HALF
    assert np.mean(got != evaluate(DIVIDE, x, n)) < 1e-5


def test_quotients_without_a_finite_result(evaluate):
    x, n = np.array([0.0, 0.0, 0.0, 3.0, 3.0, np.nan]), np.array([1.0, -2.0, 0.0, np.inf, np.nan, 1.0])
    np.testing.assert_array_equal(evaluate(QUOTIENT, x, n), evaluate(DIVIDE, x, n))
