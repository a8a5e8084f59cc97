"""The library step's FP64 functions (kpt_fast64.h) as the device evaluates
them, with the hardware's FP32 seeds, against extended precision."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CSRC = os.path.join(ROOT, "kokkos-particletransport_gb300", "csrc")
SOURCE = """
#include "kpt_fast64.h"
#define MAP(name) \\
    static __global__ void k_##name(int n, const double* x, double* y) { \\
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) \\
            y[i] = kpt_##name(x[i]); \\
    } \\
    extern "C" int t_##name(int n, const double* x, double* y) { \\
        double* d = nullptr; \\
        if (cudaMalloc(&d, 2 * sizeof(double) * n) != cudaSuccess) return 1; \\
        cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice); \\
        k_##name<<<152, 256>>>(n, d, d + n); \\
        cudaMemcpy(y, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost); \\
        cudaFree(d); \\
        return cudaGetLastError() != cudaSuccess; \\
    }
MAP(rcp) MAP(rsqrt) MAP(sqrt) MAP(cbrt) MAP(log)
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("fast64")
    src, so = str(path / "t.cu"), str(path / "t.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, src, "-o", so], check=True)
    return ctypes.CDLL(so)


def _apply(lib, name, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.empty_like(x)
    assert getattr(lib, "t_" + name)(x.size, x.ctypes.data_as(ctypes.c_void_p),
                                     y.ctypes.data_as(ctypes.c_void_p)) == 0
    return y


def _ulps(got, exact):
    return np.abs(got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact).astype(np.float64))


def _operands():
    rng = np.random.default_rng(11)
    powers = 2.0 ** np.arange(-100.0, 100.0)
    return np.concatenate([np.exp(rng.uniform(-69.0, 69.0, 200000)), rng.uniform(0.5, 8.0, 200000),
                           (powers[:, None] * rng.uniform(1.0, 2.0, 200)).ravel(), powers,
                           np.nextafter(powers[1:], 0.0), 1.0 + np.arange(1, 200) * 2.0 ** -52])


# the header's bounds: a rounded product and sum each, and the series' rest
@pytest.mark.parametrize("name,exact,bound", [
    ("rcp", lambda x: 1 / x, 1.5), ("rsqrt", lambda x: 1 / np.sqrt(x), 1.5),
    ("sqrt", np.sqrt, 1.5), ("cbrt", np.cbrt, 1.5)])
def test_algebraic_functions(lib, name, exact, bound):
    x = _operands()
    ulps = _ulps(_apply(lib, name, x), exact(x.astype(np.longdouble)))
    worst = int(ulps.argmax())
    print(name, float(ulps[worst]), x[worst])
    assert ulps[worst] <= bound


def test_cube_root_keeps_its_error_over_the_range(lib):
    """A cube root of 2^(3k) m is 2^k times that of m, bit for bit, so its error
    is that of [1, 8) everywhere."""
    m = np.random.default_rng(5).uniform(1.0, 8.0, 20000)
    want = _apply(lib, "cbrt", m)
    for k in (-33, -20, -1, 1, 11, 32):
        assert np.array_equal(_apply(lib, "cbrt", m * 2.0 ** (3 * k)), want * 2.0 ** k), k


def test_logarithm_of_draws(lib):
    rng = np.random.default_rng(12)
    n = np.concatenate([rng.integers(1, 2 ** 53, 300000, dtype=np.uint64),
                        np.arange(1, 3000, dtype=np.uint64),
                        np.uint64(2 ** 53) - np.arange(0, 3000, dtype=np.uint64)])
    u = n.astype(np.float64) * 2.0 ** -53
    exact = np.log(u.astype(np.longdouble))
    got = _apply(lib, "log", u)
    sel = exact != 0
    assert np.all(got[~sel] == 0.0)
    ulps = _ulps(got[sel], exact[sel]).max()
    print("log", float(ulps))
    assert ulps <= 2.0
