"""The fixed-point quotient and square root of the water temperature, compiled from
their header: random and edge mantissas over the exponents, and everything that is
not a normal number as the hardware has it.

Bounds in ulp: half an ulp of the final rounding plus, for the quotient, that of the
reciprocal (0.01) and of one truncated product; for the root, four truncated products
(2^-8 each at most) and the series' fourth term (2^-7.5)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble

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


def _ulp(got, ref):
    return np.abs(LD(got) - ref) / np.spacing(np.abs(ref).astype(np.float64)).astype(LD)


@pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="no wider type to compare with")
def test_rounding(run):
    rng = np.random.default_rng(3)
    m = np.concatenate([1 + rng.random(100000), 1 + np.ldexp(1.0, -np.arange(1, 53)), 2 - np.ldexp(1.0, -np.arange(1, 53))])
    a = np.ldexp(m, rng.integers(-300, 300, m.size)) * rng.choice([-1, 1], m.size)
    b = np.ldexp(rng.permutation(m), rng.integers(-300, 300, m.size))
    assert _ulp(run(0, a, b), LD(a) / LD(b)).max() < 0.52
    x = np.concatenate([np.abs(a), np.nextafter(np.ldexp(1.0, np.arange(-1000, 1000)), 0), np.ldexp(1.0, np.arange(-1000, 1000))])
    assert _ulp(run(1, x, x), np.sqrt(LD(x))).max() < 0.5 + 2.0 ** -5


def test_not_normal(run):
    v = np.array([0.0, -0.0, 1.0, -3.0, np.inf, -np.inf, np.nan, 5e-324, -1e-310, 1e308, 2.3e-308])
    a, b = (g.ravel() for g in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        want, root = a / b, np.sqrt(v)
    got = run(0, a, b)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.signbit(got[want == 0]), np.signbit(want[want == 0]))
    ok = np.isfinite(want) & (want != 0)
    assert np.array_equal(got[~ok], want[~ok], equal_nan=True)
    assert np.all(np.abs(got[ok] - want[ok]) <= np.spacing(np.abs(want[ok])))
    assert np.array_equal(run(1, v, v)[[0, 1, 4, 5, 6]], root[[0, 1, 4, 5, 6]], equal_nan=True)
    assert np.isnan(run(1, v, v)[3]) and np.all(np.abs(run(1, v, v)[7:8] - root[7:8]) <= np.spacing(root[7:8]))
