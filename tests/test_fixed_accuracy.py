"""Accuracy of the fixed-point quadrature (mpart_gb300/csrc/mpgb_fixed.cuh,
built for the host) where sums over points or small values show it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
P = ctypes.c_void_p


def _p(a):
    return a.ctypes.data_as(P)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fa") / "fa.so"
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-shared", "-fPIC", "-o", str(out),
                    os.path.join(HERE, "fixed_accuracy_harness.cpp")], check=True)
    return ctypes.CDLL(str(out))


@pytest.mark.parametrize("expr", [0, 1])
@pytest.mark.parametrize("x,abs_tol", [(4.0, 1e-17), (1.0, 5e-18), (30.0, 1e-22), (1.0, 1e-16), (1.0, 0.9e-15), (3.0, 3e-15),
                                       (0.5, 1e-12), (1e-300, 1e-15)])
def test_tight_absolute_tolerances(lib, expr, x, abs_tol):
    """relTol = 0: a threshold absTol / |x_D| below 2^-50 is left to FP64 (5e-18
    at x_D = 1 took all of 2^22 intervals here, 255 there); above it the integral
    ends far below the budget, with the node values' 2^-55, the polynomial's and
    the sums' few 2^-58: 2^-53 (Exp: of the integral).  (The subdivision goes to
    differences of 2^-50: its own error is below that.)"""
    r = np.random.default_rng(3)
    out = np.zeros(2)
    for _ in range(20):
        b = np.ascontiguousarray(r.normal(0.0, 0.5, 6))
        lib.fa_tight(expr, _p(b), ctypes.c_double(x), ctypes.c_double(abs_tol), _p(out))
        if abs_tol / x < 2.0 ** -50:
            assert out[0] == 0
        else:
            assert 0 < out[0] <= 2 ** 13
            assert out[1] <= 2.0 ** -53 + abs_tol / x


@pytest.mark.parametrize("expr", [0, 1])
def test_hermite_function_moments_have_no_common_bias(lib, expr):
    """The moments' errors average out over points, up to the envelope's order
    4 and beyond: those of Hermite functions meet in alternating sums, where a
    common 6e-17 of the fifth came back as 1e-15 of an order-5 gradient.  A
    moment's error is some 4e-16 at worst (j = 5, over these points): the mean
    of 40,000 is within 4 x 4e-16 / 200 = 8e-18, and the functions' own
    2^-57 = 7e-18 on top."""
    r = np.random.default_rng(17 + expr)
    n = 40_000
    x = np.where(np.arange(n) % 2 == 0, r.standard_normal(n), r.standard_normal(n) ** 2 + 0.5 * r.standard_normal(n))
    x = np.where(np.abs(x) < 1e-3, 1e-3, x)
    b = r.normal(0.0, 0.1, (n, 6)) * np.sign(x)[:, None] ** np.arange(6) * np.abs(x)[:, None] ** np.arange(6)
    b *= np.minimum(1.0, 25.0 / np.abs(b).sum(1))[:, None]
    a = 0.5 + 0.05 * r.standard_normal(n)
    mean = np.zeros(6)
    lib.fa_moment_bias(expr, _p(b), _p(a), _p(x), ctypes.c_long(n), ctypes.c_double(1e-7), _p(mean))
    assert np.all(np.abs(mean) <= 1.5e-17), mean


@pytest.mark.parametrize("budget", [1, 2, 17])
def test_intervals_of_an_exhausted_budget(lib, budget):
    """The count is the next call's sort key, also where the budget ended it."""
    assert lib.fa_over(budget) == budget
