"""What the fixed-point functions rest on, compiled from their headers: the reciprocal
and the root over every leading 24 bits (the single-precision seeds must err to one
side, since an unsigned remainder would wrap), exp(-x) beside 1, and the temperature
terms over the climate and past its ends.

Bounds, from the error terms. Reciprocal of a mantissa, units of 2^-64: at most 16 for
e^3 with e below 2^-20, 4 for the leading bits of e in its square, 6 for truncations, all
low, and 2 high for a truncated e. exp_neg below 2^-8: 2 units of 2^-64 beside the last
rounding; above it exp's own 2^-4 ulp. rlh and apt: the last rounding and 2^-54 for the
exponent's truncations, below 2^-52. lwt, whose emissivity changes sign: its five high
products are 7 units low of 2^50 or more units of the emissivity 0.02 at the coldest,
which is 2 units of 2^-52 of the terms' scale, 0.281; elsewhere less."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble
needs_quad = pytest.mark.skipif(np.finfo(LD).nmant < 63, reason="no wider type to compare with")
SRC = r"""
#include <cuda_runtime.h>
#include "wg_radiation.cuh"
using wg::fm::u64;
using wg::fm::TempTerms;
// f 0: worst and best (2^127 / m) - rcp_mant(m); f 1: roots that differ from the FP64 ones
__global__ void k_all(int f, unsigned long long low, long long *o) {
  const unsigned lead = blockIdx.x * blockDim.x + threadIdx.x;   // 2^23 of them
  const u64 m = (1ull << 63) | ((u64)lead << 40) | low;
  if (f == 0) {
    const __int128 rest = ((__int128)1 << 127) - (__int128)((unsigned __int128)m * wg::fm::rcp_mant(m));
    const long long d = (long long)(rest >= 0 ? rest / m : -((-rest + m - 1) / m));
    atomicMax(o, d);
    atomicMin(o + 1, d);
  } else {
    for (unsigned e = 1022; e < 1024; ++e) {
      const double x = wg::fm::double_of((m << 1 >> 12) | ((u64)e << 52));
      if (wg::fm::bits_of(wg::fm::sqrt(x)) != wg::fm::bits_of(::sqrt(x))) atomicAdd((unsigned long long *)o, 1ull);
    }
  }
}
__global__ void k(int f, const double *x, double *o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (f == 0) { o[i] = wg::fm::exp_neg(x[i]); return; }
  const TempTerms t = wg::fm::temp_terms((float)x[i]);
  o[i] = t.rlh;
  o[n + i] = t.apt;
  o[2 * n + i] = t.lwt;
}
extern "C" int all(int f, unsigned long long low, long long *o) {
  long long *d = nullptr;
  if (cudaMalloc(&d, 16)) return 1;
  cudaMemcpy(d, o, 16, cudaMemcpyHostToDevice);
  k_all<<<(1 << 23) / 256, 256>>>(f, low, d);
  const int e = (int)cudaMemcpy(o, d, 16, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
extern "C" int run(int f, const unsigned long long *e2, const unsigned long long *l2, const double *x, double *o, int n) {
  cudaMemcpyToSymbol(wg::fm::g_exp2_tab, e2, sizeof(wg::fm::g_exp2_tab));
  cudaMemcpyToSymbol(wg::fm::g_log2_tab, l2, sizeof(wg::fm::g_log2_tab));
  double *d = nullptr;
  const size_t b = (size_t)n * sizeof(double);
  if (cudaMalloc(&d, 4 * b)) return 1;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(f, d, d + n, n);
  const int e = (int)cudaMemcpy(o, d + n, (f ? 3 : 1) * b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from watergap2_gb300 import build
    d = tmp_path_factory.mktemp("seeds")
    (d / "s.cu").write_text(SRC)
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(os.path.dirname(build.__file__), "csrc"), "-o", str(d / "s.so"),
                    str(d / "s.cu")], check=True)
    return ctypes.CDLL(str(d / "s.so"))


LOW = [0, (1 << 40) - (1 << 11)]   # the 40 bits below the leading 24: least and most of a double's


@pytest.mark.parametrize("low", LOW)
def test_reciprocals_of_all_leading_bits(lib, low):
    o = np.array([-2 ** 62, 2 ** 62], np.int64)
    assert lib.all(0, ctypes.c_ulonglong(low), o.ctypes.data_as(ctypes.c_void_p)) == 0
    assert -2 <= o[1] and o[0] <= 26


@pytest.mark.parametrize("low", LOW)
def test_roots_of_all_leading_bits(lib, low):
    o = np.zeros(2, np.int64)
    assert lib.all(1, ctypes.c_ulonglong(low), o.ctypes.data_as(ctypes.c_void_p)) == 0
    assert o[0] == 0


def _call(lib, f, x):
    x = np.ascontiguousarray(x, np.float64)
    e2 = np.array([int(np.rint(np.exp2(LD(j) / 256) * LD(2) ** 63)) for j in range(256)], np.uint64)
    out = np.empty((3 if f else 1, x.size))
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (e2, np.zeros(512, np.uint64), x, out)]   # (no logarithms here)
    assert lib.run(f, *ptr, x.size) == 0
    return out


@needs_quad
def test_exp_neg(lib):
    small = np.concatenate([np.logspace(-320, np.log10(2.0 ** -8), 4000)[:-1], np.linspace(1e-3, 2.0 ** -8, 4000)[:-1],
                            [5e-324, 2.0 ** -54, 2.0 ** -53, 2.0 ** -30, np.nextafter(2.0 ** -8, 0)]])
    large = np.concatenate([np.linspace(2.0 ** -8, 31.9, 4000), [2.0 ** -8, np.nextafter(2.0 ** -8, 1)]])
    for x, bound in ((small, 0.5 + 2.0 ** -9), (large, 0.5 + 2.0 ** -4)):
        ref = np.exp(-LD(x))
        ulp = np.spacing(np.nextafter(ref.astype(np.float64), 0)).astype(LD)   # below a power of two: the ulp there
        assert (np.abs(LD(_call(lib, 0, x)[0]) - ref) / ulp).max() < bound
    with np.errstate(all="ignore"):
        x = np.array([0., -0., np.inf, -1., np.nan, 746.])
        got = _call(lib, 0, x)[0]
    assert np.array_equal(got[[0, 1, 2, 5]], [1., 1., 0., 0.]) and abs(got[3] - np.e) < 1e-15 and np.isnan(got[4])


def _terms(T):
    T = LD(T)
    rlh = 1 / np.where(T > 0, LD(2.501) - LD(0.002361) * T, LD(2.835))
    s = LD(4098.) * LD(0.6108) * np.exp(LD(17.27) * T / (T + LD(237.3))) / (T + LD(237.3)) ** 2
    scale = LD(0.000000004903) * (T + LD(273.2)) ** 4 * rlh
    return rlh, s / (s + LD(0.0016286 * 101.3) * rlh), (LD(0.261) * np.exp(LD(-0.000777) * T * T) - LD(0.02)) * scale, scale


@needs_quad
def test_temperature_terms(lib):
    rng = np.random.default_rng(1)
    edge = np.float32([0, 1e-30, 1e-7, 57.4979, 127.99999])
    T = np.concatenate([rng.uniform(-128, 128, 200000).astype(np.float32)[1:], edge, -edge, np.arange(-127, 128, dtype=np.float32),
                        np.float32(57.498) + np.arange(-2000, 2000) * np.spacing(np.float32(57.498))]).astype(np.float32)
    T = T[np.abs(T) < 128]
    rlh, apt, lwt, scale = _terms(T)
    got = LD(_call(lib, 1, T))
    ulp = LD(2.0) ** -52
    assert (np.abs(got[0] - rlh) / rlh).max() < ulp
    assert (np.abs(got[1] - apt) / apt).max() < ulp
    assert (np.abs(got[2] - lwt) / (LD(0.281) * scale)).max() < 2 * ulp


@needs_quad
def test_temperature_terms_past_the_climate(lib):
    T = np.concatenate([np.linspace(128, 200, 100), -np.linspace(128, 200, 100)]).astype(np.float32)
    rlh, apt, lwt, scale = _terms(T)
    got = LD(_call(lib, 1, T))
    few = LD(2.0) ** -52 * 64   # FP64 expressions, an exponent of up to 92
    assert (np.abs(got[0] - rlh) / rlh).max() < few
    assert (np.abs(got[1] - apt) / apt).max() < 4 * few
    assert (np.abs(got[2] - lwt) / scale).max() < few
    rlh, apt, lwt = _call(lib, 1, np.array([np.nan]))[:, 0]
    assert np.isnan([apt, lwt]).all() and abs(rlh - 1 / 2.835) < 1e-16   # the latent heat tests T > 0
