"""The fixed-point quadrature (mpart_gb300/csrc/mpgb_fixed.cuh), built for the
host: its exponential, logarithm and reciprocal against 40-digit decimals, its
traversal and moments against the same rule in long double over both
rectifiers, both forms of the integrand, both rules and forced subdivision,
and the tables equal to what their generator writes.

Tolerances: a handful of truncations at 2^-57 (node values) and 2^-62
(moments), so 2^-55 per node; an integral adds its polynomial's six steps at
2^-58 and half a unit of 2^-57 per accepted interval: 2^-53, the spacing of a
double near 1."""
import ctypes
import os
import subprocess
import sys
from decimal import Decimal, getcontext

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "mpart_gb300", "csrc")
P = ctypes.c_void_p


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fx") / "fx.so"
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-shared", "-fPIC", "-o", str(out),
                    os.path.join(HERE, "fixed_harness.cpp")], check=True)
    return ctypes.CDLL(str(out))


def _points():
    r = np.random.default_rng(4)
    edges = np.array([0.0, 2.0 ** -58, -2.0 ** -58, 31.0, -31.0, np.log(2.0), -np.log(2.0), 1e-300])
    x = np.concatenate([edges, r.uniform(-31, 31, 1500), r.normal(0, 1, 1500)])
    return np.trunc(x * 2.0 ** 58) / 2.0 ** 58  # representable: only the functions' own error is seen


def test_softplus_and_exp(lib):
    getcontext().prec = 40
    x = _points()
    n = x.size
    g, gp, m, E = np.zeros(2 * n), np.zeros(2 * n), np.zeros(2 * n), np.zeros(n, np.int32)
    lib.fx_softplus(x.ctypes.data_as(P), g.ctypes.data_as(P), gp.ctypes.data_as(P), ctypes.c_long(n))
    lib.fx_exp(x.ctypes.data_as(P), m.ctypes.data_as(P), E.ctypes.data_as(P), ctypes.c_long(n))
    tol = Decimal(2) ** -55
    for i in range(n):
        d = Decimal(float(x[i]))
        e = (-abs(d)).exp()
        val = lambda a: Decimal(float(a[2 * i])) + Decimal(float(a[2 * i + 1]))  # noqa: E731
        assert abs(val(g) - ((1 + e).ln() + max(d, Decimal(0)))) <= tol
        assert abs(val(gp) - (1 / (1 + e) if d > 0 else e / (1 + e))) <= tol
        assert abs(val(m) * Decimal(2) ** int(E[i]) / d.exp() - 1) <= tol


@pytest.mark.parametrize("expr", [0, 1])
@pytest.mark.parametrize("env", [0, 1])
@pytest.mark.parametrize("simpson,tol,min_sub", [(0, 1e-6, 0), (1, 1e-8, 0), (0, 1e-6, 2)])
def test_integrals_match_long_double(lib, expr, env, simpson, tol, min_sub):
    r = np.random.default_rng(10 * expr + env)
    out = np.zeros(4)
    done = 0
    for it in range(150):
        b = r.normal(0, np.exp(r.normal(0, 1)), 6)
        a, Z, xd = (r.normal(0, 1), abs(8 * r.normal() * r.normal()), abs(r.normal()) + 1e-3)
        if it % 7 == 0:
            Z *= 40.0  # beyond 126: the envelope's coarser exponent format
        if it % 10 == 0:
            b[1:] = 0.0  # constant integrand: one interval
        if abs(b).sum() + abs(a) > 31 or b[0] < -4 or Z > 1900:
            continue
        lib.fx_integrate(expr, env, b.ctypes.data_as(P), ctypes.c_double(a), ctypes.c_double(Z), ctypes.c_double(xd),
                         ctypes.c_double(tol), simpson, min_sub, out.ctypes.data_as(P))
        assert out[2] == out[3]
        assert out[0] <= 2.0 ** -53 and out[1] <= 2.0 ** -53
        done += 1
    assert done > 100


def test_tables_match_their_generator():
    out = subprocess.run([sys.executable, os.path.join(CSRC, "gen_fixed_tables.py")], check=True,
                         capture_output=True, text=True).stdout
    with open(os.path.join(CSRC, "mpgb_fixed_tables.h")) as f:
        assert f.read() == out
