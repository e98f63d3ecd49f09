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
