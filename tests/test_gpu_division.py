"""The corrected quotients and reciprocals of the row kernels (ufe_internal.h) against the host's IEEE
division, bit for bit (run with -m gpu): random operands, all-ones and near-all-ones significands,
exponents on both sides of the windows in which the short forms are taken, zeros, subnormals, infinities
and NaN. The parity sweeps and the boundary means rely on these quotients being the IEEE ones."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from ufemism_gb300 import api, build

pytestmark = pytest.mark.gpu

SOURCE = """
#include <cuda_runtime.h>
#include "%s/ufe_internal.h"
namespace ufe {
__global__ void k_ops(int op, int n, const double *a, const double *b, double *o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = op == 0 ? divide_by(a[i], b[i], 1.0 / b[i])
         : op == 1 ? reciprocal_rn(b[i])
         : op == 2 ? divide_by(a[i], b[i], reciprocal_rn(b[i]))
                   : reciprocal_newton(b[i]);
}
}
extern "C" int run(int op, int n, const double *a, const double *b, double *o) {
  double *d = nullptr;
  cudaError_t e = cudaMalloc(&d, 3 * (size_t)n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(d, a, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) ufe::k_ops<<<(n + 255) / 256, 256>>>(op, n, d, d + n, d + 2 * (size_t)n);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(o, d + 2 * (size_t)n, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  if (d) cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    api.init(0)
    d = tmp_path_factory.mktemp("division")
    src, lib = os.path.join(d, "ops.cu"), os.path.join(d, "ops.so")
    with open(src, "w") as f:
        f.write(SOURCE % build.SRC)
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared",
                    "-cudart", "static", "-o", lib, src], check=True, capture_output=True)
    L = ct.CDLL(lib)

    def call(op, a, b):
        a, b = np.ascontiguousarray(a, dtype=np.float64), np.ascontiguousarray(b, dtype=np.float64)
        o = np.empty(b.size)
        assert L.run(op, b.size, *(ct.c_void_p(x.ctypes.data) for x in (a, b, o))) == 0
        return o

    return call


def operands(kind, rng, n=400000):
    def number(significand, low, high):
        s = np.ldexp(significand.astype(np.float64), -52)
        return np.ldexp(s, rng.integers(low, high, s.size)) * rng.choice([-1.0, 1.0], s.size)

    full = rng.integers(2**52, 2**53, (2, n))
    if kind == "random":
        return number(full[0], -60, 60), number(full[1], -60, 60)
    if kind == "ones":       # the significands for which the last step alone would not do, and their neighbours
        return number(full[0], -60, 60), number(2**53 - 1 - rng.integers(0, 4, n), -60, 60)
    if kind == "low":
        return number(2**52 + rng.integers(0, 64, n), -60, 60), number(2**52 + rng.integers(0, 64, n), -60, 60)
    if kind == "counts":
        return number(full[0], -60, 60), rng.integers(1, 33, n).astype(np.float64)
    if kind == "windows":    # biased exponents 200 and 1800 are 2^-823 and 2^777
        a = np.concatenate([number(full[0, :n // 2], -826, -820), number(full[0, n // 2:], 773, 780)])
        return a, number(full[1], -4, 4)
    if kind == "quotients":  # the quotient leaves the window, the operands do not
        return number(full[0], 300, 770), number(full[1], -520, -1)
    if kind == "divisors":
        b = np.concatenate([number(full[1, :n // 2], -826, -820), number(full[1, n // 2:], 773, 780)])
        return number(full[0], -60, 60), b
    if kind == "wide":
        return number(full[0], -1021, 1023), number(full[1], -1021, 1022)
    special = np.array([0.0, -0.0, 5e-324, -5e-324, 2.0**-1022, 2.0**-1022 - 5e-324, np.inf, -np.inf, np.nan, 1.0, 3.0, -7.0,
                        1.7976931348623157e308, 1e-300, 1e300, 2.0 - 2.0**-52])
    a, b = np.meshgrid(special, special)
    return a.ravel(), b.ravel()


def same_bits(x, y):
    both_nan = np.isnan(x) & np.isnan(y)
    return np.all(both_nan | (x.view(np.int64) == y.view(np.int64)))


@pytest.mark.parametrize("kind", ["random", "ones", "low", "counts", "windows", "quotients", "divisors", "wide", "special"])
def test_rounded_as_the_division(device, kind):
    a, b = operands(kind, np.random.default_rng(17))
    with np.errstate(all="ignore"):
        quotient, reciprocal = a / b, 1.0 / b
    assert same_bits(device(0, a, b), quotient)
    assert same_bits(device(1, a, b), reciprocal)
    assert same_bits(device(2, a, b), quotient)
    if kind in ("random", "ones", "low", "counts"):   # to within a unit in the last place
        y = device(3, a, b)
        assert np.all(np.abs(y.view(np.int64) - reciprocal.view(np.int64)) <= 1)
