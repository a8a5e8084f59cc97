"""The library step's FP64 functions (kpt_fast64.h), host build: error bounds
against extended precision over the operands the solver meets and the ends of
the fast range, and the fall-backs beyond it."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc")
SOURCE = """
#include "kpt_fast64.h"
#define MAP(name) extern "C" void t_##name(int n, const double* x, double* y) { \\
    for (int i = 0; i < n; ++i) y[i] = kpt_##name(x[i]); }
MAP(rcp) MAP(rsqrt) MAP(sqrt) MAP(cbrt) MAP(log)
extern "C" void t_sincos(int n, const uint64_t* u, double* s, double* c) {
    for (int i = 0; i < n; ++i) kpt_sincos_turn(u[i], s + i, c + i); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("fast64")
    src, so = str(path / "t.cpp"), str(path / "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, src, "-o",
                    so], check=True)
    return ctypes.CDLL(so)


def _apply(lib, name, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.empty_like(x)
    getattr(lib, "t_" + name)(x.size, x.ctypes.data_as(ctypes.c_void_p),
                              y.ctypes.data_as(ctypes.c_void_p))
    return y


def _ulps(got, exact):
    """Error in units of the last place of the result (exact: extended precision)."""
    return np.abs(got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact).astype(np.float64))


def _operands():
    rng = np.random.default_rng(11)
    x = [np.exp(rng.uniform(-69.0, 69.0, 200000)), rng.uniform(0.5, 4.0, 200000),
         2.0 ** np.arange(-100.0, 100.0), np.nextafter(2.0 ** np.arange(-99.0, 100.0), 0.0),
         1.0 + np.arange(1, 200) * 2.0 ** -52]
    return np.concatenate(x)


@pytest.mark.parametrize("name,exact,bound", [
    ("rcp", lambda x: 1 / x, 1.5), ("rsqrt", lambda x: 1 / np.sqrt(x), 1.5),
    ("sqrt", np.sqrt, 1.5), ("cbrt", np.cbrt, 1.5)])
def test_algebraic_functions(lib, name, exact, bound):
    x = _operands()
    assert _ulps(_apply(lib, name, x), exact(x.astype(np.longdouble))).max() <= bound


def test_logarithm_of_draws(lib):
    rng = np.random.default_rng(12)
    n = np.concatenate([rng.integers(1, 2 ** 53, 300000, dtype=np.uint64),
                        np.arange(1, 3000, dtype=np.uint64),
                        np.uint64(2 ** 53) - np.arange(0, 3000, dtype=np.uint64)])
    u = n.astype(np.float64) * 2.0 ** -53
    exact = np.log(u.astype(np.longdouble))
    got = _apply(lib, "log", u)
    assert np.all(got[exact == 0] == 0.0)
    sel = exact != 0
    assert _ulps(got[sel], exact[sel]).max() <= 2.0


def test_sine_and_cosine_of_draws(lib):
    rng = np.random.default_rng(13)
    edges = np.concatenate([k * 2 ** 50 + np.arange(-3, 4) for k in range(1, 8)])
    n = np.concatenate([rng.integers(0, 2 ** 53, 300000), edges, np.arange(0, 50),
                        2 ** 53 - np.arange(1, 50)]).astype(np.uint64)
    s, c = np.empty(n.size), np.empty(n.size)
    lib.t_sincos(n.size, *(a.ctypes.data_as(ctypes.c_void_p) for a in (n, s, c)))
    # the angle reduced exactly to [-1/8, 1/8] of a turn, then extended precision
    q = (n + np.uint64(2 ** 50)) // np.uint64(2 ** 51)
    f = (n.astype(np.int64) - q.astype(np.int64) * 2 ** 51).astype(np.longdouble) / 2 ** 53
    pi = np.longdouble("3.14159265358979323846264338327950288")
    es, ec = np.sin(2 * pi * f), np.cos(2 * pi * f)
    quarter = (q % np.uint64(4)).astype(int)
    es, ec = (np.choose(quarter, [es, ec, -es, -ec]), np.choose(quarter, [ec, -es, -ec, es]))
    # half an ulp of 1 for the rounding, a quarter for the cut polynomial
    assert np.abs(s - es).max() <= 0.75 * 2.0 ** -52
    assert np.abs(c - ec).max() <= 0.75 * 2.0 ** -52


def test_operands_beyond_the_fast_range(lib):
    x = np.array([0.0, 1e-310, 1e-200, 1e200, np.inf, -2.0, np.nan])
    with np.errstate(all="ignore"):
        for name, f in (("rcp", lambda v: 1 / v), ("sqrt", np.sqrt), ("cbrt", np.cbrt),
                        ("rsqrt", lambda v: 1 / np.sqrt(v))):
            # the C library's functions, a few ulp apart between libraries
            np.testing.assert_allclose(_apply(lib, name, x), f(x), rtol=1e-15, equal_nan=True)
