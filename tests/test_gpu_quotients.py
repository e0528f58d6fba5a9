"""The fixed-point quotient and square root of the water temperature, compiled from
their header: random and edge mantissas over the exponents, and everything that is
not a normal number as the hardware has it. Both round correctly, so the
results are the bits of the host's."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "wg_fastmath.cuh"
__global__ void k(int f, const double *x, const double *y, double *o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) o[i] = f ? wg::fm::sqrt(x[i]) : wg::fm::div(x[i], y[i]);
}
extern "C" int run(int f, const double *x, const double *y, double *o, int n) {
  double *d = nullptr;
  const size_t b = (size_t)n * sizeof(double);
  if (cudaMalloc(&d, 3 * b)) return 1;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(f, d, d + n, d + 2 * (size_t)n, n);
  const int e = (int)cudaMemcpy(o, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from watergap2_gb300 import build
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(os.path.dirname(build.__file__), "csrc"), "-o", str(d / "q.so"),
                    str(d / "q.cu")], check=True)
    lib = ctypes.CDLL(str(d / "q.so"))

    def call(f, x, y):
        x, y = (np.ascontiguousarray(v, np.float64) for v in (x, y))
        out = np.empty_like(x)
        ptr = [v.ctypes.data_as(ctypes.c_void_p) for v in (x, y, out)]
        assert lib.run(f, *ptr, len(x)) == 0
        return out
    return call


def test_rounding(run):
    rng = np.random.default_rng(3)
    m = np.concatenate([1 + rng.random(100000), 1 + np.ldexp(1.0, -np.arange(1, 53)), 2 - np.ldexp(1.0, -np.arange(1, 53))])
    a = np.ldexp(m, rng.integers(-300, 300, m.size)) * rng.choice([-1, 1], m.size)
    b = np.ldexp(rng.permutation(m), rng.integers(-300, 300, m.size))
    assert np.array_equal(run(0, a, b), a / b)
    x = np.concatenate([np.abs(a), np.nextafter(np.ldexp(1.0, np.arange(-1000, 1000)), 0), np.ldexp(1.0, np.arange(-1000, 1000))])
    assert np.array_equal(run(1, x, x), np.sqrt(x))


def test_not_normal(run):
    v = np.array([0.0, -0.0, 1.0, -3.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 1e308, 2.3e-308])
    a, b = (g.ravel() for g in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        want, root = a / b, np.sqrt(v)
    got = run(0, a, b)
    assert np.array_equal(got, want, equal_nan=True) and np.array_equal(np.signbit(got[want == 0]), np.signbit(want[want == 0]))
    assert np.array_equal(run(1, v, v), root, equal_nan=True)
