"""
The Boys table of the integral kernels (csrc/hf_boys.h, compiled here for the
host: the same table, the same arithmetic) against F_n in 50 digits: every
order that a kernel reads, x = 0, both sides of every interval edge and of the
table's end 36 + 3N, interval middles, and far beyond.

Bound: the table's coefficients, seven fused steps and the downward recursion
round by some 1e-15 in all (relative); 3e-15, half of it for the closed form's
products beyond the table.
"""

from __future__ import annotations

import ctypes
import os
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

from conftest import ROOT

MAX_N = 6
SHIM = """
#include "hf_boys.h"
static const std::vector<double> table = hf::make_boys_tables();
template <int L> static void run(int n, const double* x, double a, double scale, double* out) {
    const hf::BoysShared b{table.data() + hf::boys_offset(L)};
    for (int i = 0; i < n; ++i) {
        double g[L + 1];
        b.operator()<L>(a, x[i], scale, g);
        for (int k = 0; k <= L; ++k) out[i * (L + 1) + k] = g[k];
    }
}
extern "C" int max_order() { return hf::BOYS_MAX_N; }
extern "C" void boys(int L, int n, const double* x, double a, double scale, double* out) {
    switch (L) {
        case 0: return run<0>(n, x, a, scale, out);
        case 1: return run<1>(n, x, a, scale, out);
        case 2: return run<2>(n, x, a, scale, out);
        case 3: return run<3>(n, x, a, scale, out);
        case 4: return run<4>(n, x, a, scale, out);
        case 5: return run<5>(n, x, a, scale, out);
        case 6: return run<6>(n, x, a, scale, out);
    }
}
"""


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    d = tmp_path_factory.mktemp("boys")
    src, lib = d / "shim.cpp", d / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-Wno-unknown-pragmas",
                    "-I", os.path.join(ROOT, "ab-initio-md_b200", "csrc"), str(src), "-o", str(lib)], check=True)
    so = ctypes.CDLL(str(lib))
    dp = ctypes.POINTER(ctypes.c_double)
    so.boys.argtypes = [ctypes.c_int, ctypes.c_int, dp, ctypes.c_double, ctypes.c_double, dp]
    assert so.max_order() == MAX_N

    def run(L, x, a=-0.5, scale=1.0):       # (-2a)^n = 1
        x = np.ascontiguousarray(x, dtype=float)
        out = np.empty((x.size, L + 1))
        so.boys(L, x.size, x.ctypes.data_as(dp), a, scale, out.ctypes.data_as(dp))
        return out
    return run


def _exact(top, x):
    """F_0 .. F_top(x) in 50 digits: the ascending series and downward recursion, or erfc(sqrt x) = 0 and upward."""
    x = Decimal(float(x))
    ex = (-x).exp()
    F = [Decimal(0)] * (top + 1)
    if x < 130:                                     # erfc(sqrt 130) < 1e-57
        term = Decimal(1) / (2 * top + 1)
        s, k = term, 1
        while term > s * Decimal(10) ** -45:
            term *= 2 * x / (2 * top + 2 * k + 1)
            s += term
            k += 1
        F[top] = ex * s
        for n in range(top - 1, -1, -1):
            F[n] = (2 * x * F[n + 1] + ex) / (2 * n + 1)
    else:
        pi = Decimal("3.14159265358979323846264338327950288419716939937511")
        F[0] = (pi / x).sqrt() / 2
        for n in range(top):
            F[n + 1] = ((2 * n + 1) * F[n] - ex) / (2 * x)
    return np.array([float(f) for f in F])


@pytest.mark.parametrize("L", range(MAX_N + 1))
def test_table(table, L):
    getcontext().prec = 50
    end = 36 + 3 * L
    edges = np.arange(0, 8 * end + 1) / 8.0
    x = np.concatenate([edges, np.nextafter(edges, np.inf), np.nextafter(edges[1:], 0.0), edges + 1.0 / 16,
                        end + np.geomspace(1e-9, 264.0, 40), [1e3, 1e5, 1e8]])
    got = table(L, x)
    ref = np.array([_exact(L, v) for v in x])
    assert (np.abs(got - ref) <= 3e-15 * ref).all(), np.max(np.abs(got / ref - 1))


@pytest.mark.parametrize("L", range(MAX_N + 1))
def test_factors(table, L):
    """scale (-2 alpha)^n F_n, and NaN through both branches' test."""
    x = np.array([0.0, 0.3, 7.7, 35.9, 60.0])
    ratio = table(L, x, 0.7, 3.0) / table(L, x)
    assert np.abs(ratio / (3.0 * (-1.4) ** np.arange(L + 1)) - 1).max() <= 4e-15
    assert np.isnan(table(L, [np.nan])).all()
